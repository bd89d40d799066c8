// tdse_ground.cu -- the ground state of a grid with its vectors in the shared memory of a small cluster.
//
// build_grids_kernel iterates one grid per CTA with its vectors in L2: 8.1 ms for 8001 sites, where a
// pass waits for L2 at every site.  Few grids (a single call builds one) take a cluster each instead.
// The iteration stops on rounding noise (CV is 1e-15), so psi0 depends on the order of every sum in
// the twelfth digit, and complex64 propagation on its last bit: the 256 chunks, the scans and the
// sums are those of ground_state(), operation by operation, and so is the result, bit for bit.
//
// Eight CTAs hold a warp of chunks each, so that every warp has its own FP64 units; three more warps
// per CTA share what is independent per site, the normalising division and the quotient's terms (three
// divisions by 12), which are 60 of the 75 FP64 instructions of a site.  What is left is FP64 issue and
// six cluster barriers an iteration.  8001 sites, 42 iterations: 8.1 -> 2.15 ms; 601 sites, 46
// iterations: 1.1 -> 0.51 ms.  (Finer chunks over sixteen CTAs took 0.42 and 0.30 ms, but their sums
// stop the iteration elsewhere: psi0 moved by 1e-11.)
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "launch.cuh"
#include "tdse_host.cuh"
#include "tdse_solver.cuh"
#include "tdse_step.cuh"

namespace mma {
namespace {

namespace cg = cooperative_groups;

constexpr int kVectors = 9;  // ib12, h, F, g, G, V, psi, y, M2 psi
constexpr int kNC = 8;       // CTAs: one warp of the 256 threads each
constexpr int kT = 32, kSub = 4;  // its lanes, and the warps that share its per-site work
static_assert(kNC * kT == kThreads, "one warp of chunks per CTA");

// What crosses CTAs: per warp the scans' maps and the partial sums, and the neighbours' edge sites.
struct Shared {
    double cf[kWarps], bf[kWarps], cb[kWarps], bb[kWarps];
    double norm[kWarps], quot[kWarps * 2];
    double left, right;  // psi before this CTA's first site and past its last
};

__global__ void __launch_bounds__(kT* kSub) ground_state_cluster_kernel(const mma_tdse_grid* grids, int m_cap)
{
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), w = rank, lane = threadIdx.x & 31, sub = threadIdx.x >> 5;
    const int t = rank * kT + lane;
    extern __shared__ __align__(16) double vec[];
    __shared__ Shared S;
    const int LV = m_cap * kT;
    double *const ib = vec, *const hh = ib + LV, *const FF = hh + LV, *const gg = FF + LV, *const GG = gg + LV,
                 *const vq = GG + LV, *const psi = vq + LV, *const yl = psi + LV, *const mq = yl + LV;

    const mma_tdse_grid G = grids[blockIdx.x / kNC];
    const int64_t n = G.n, L = G.m * kThreads;
    const int m = (int)G.m;
    const double* const tab = G.gs_tab;
    auto pot = [&](int64_t j) { return j >= 0 && j < n ? G.gv[j] : 0.0; };  // V, left there by the table build
    for (int i = sub; i < m; i += kSub) {
        const int64_t j = (int64_t)t * m + i, e = (int64_t)i * kThreads + t;
        const int q = i * kT + lane;
        ib[q] = tab[GS_IB12 * L + e];
        hh[q] = tab[GS_H * L + e];
        FF[q] = tab[GS_F * L + e];
        gg[q] = tab[GS_G * L + e];
        GG[q] = tab[GS_GG * L + e];
        vq[q] = pot(j);
        psi[q] = j < n ? 1.0 : 0.0;  // tools.c:39-42
    }
    const double vl = pot((int64_t)t * m - 1), vr = pot((int64_t)(t + 1) * m);
    if (threadIdx.x == 0 && rank == 0) S.left = 0.0;
    if (threadIdx.x == 0 && rank == kNC - 1) S.right = 0.0;
    cluster.sync();  // every CTA has started: its shared memory may be written
    const int last = (m - 1) % kSub;  // the warp that writes site m - 1
    auto send_edges = [&] {
        if (lane == 0 && sub == 0 && rank > 0) cluster.map_shared_rank(&S, rank - 1)->right = psi[0];
        if (lane == 31 && sub == last && rank + 1 < kNC)
            cluster.map_shared_rank(&S, rank + 1)->left = psi[(m - 1) * kT + 31];
    };
    send_edges();
    cluster.sync();
    const double inv_dx2 = 1.0 / (G.dx * G.dx);
    double e_old = G.Eguess, energy = G.Eguess, test = 0.0;
    int64_t it = 0;
    int status = MMA_OK;
    for (;;) {
        // ---- solve (K - Eg M2) res = M2 psi: the sweeps of one warp, scan_forward and scan_backward
        // with the warps' maps through every CTA's shared memory
        double c = 0.0, b = 0.0;
        if (sub == 0) {
            double pm = lane == 0 ? S.left : psi[(m - 1) * kT + lane - 1];
            const double nx = lane == 31 ? S.right : psi[lane + 1];
            double pc = psi[lane], yprev = 0.0;
            for (int i = 0; i < m; i++) {
                const int q = i * kT + lane;
                const double pn = i + 1 < m ? psi[q + kT] : nx;
                const double r = fma(10.0, pc, pm + pn);
                const double y = fma(-hh[q], yprev, ib[q] * r);
                yl[q] = y;
                yprev = y;
                pm = pc;
                pc = pn;
            }
            c = FF[(m - 1) * kT + lane];
            b = yprev;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const double cp = shfl_up(c, d), bp = shfl_up(b, d);
                if (lane >= d) {
                    b = axpy_(c, bp, b);
                    c = mul_(c, cp);
                }
            }
            const double cl = shfl_idx(c, 31), bl = shfl_idx(b, 31);
            if (lane < kNC) {
                Shared* const R = cluster.map_shared_rank(&S, lane);
                R->cf[w] = cl;
                R->bf[w] = bl;
            }
        }
        cluster.sync();
        if (sub == 0) {
            double yin = 0.0;
            for (int q = 0; q < w; q++) yin = axpy_(S.cf[q], yin, S.bf[q]);
            {
                const double cp = shfl_up(c, 1), bp = shfl_up(b, 1);
                yin = lane == 0 ? yin : axpy_(cp, yin, bp);
            }
            double unext = 0.0;
            for (int i = m - 1; i >= 0; i--) {
                const int q = i * kT + lane;
                const double y = fma(FF[q], yin, yl[q]);
                const double u = fma(-gg[q], unext, y);
                yl[q] = u;
                unext = u;
            }
            c = GG[lane];
            b = unext;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const double cp = shfl_down(c, d), bp = shfl_down(b, d);
                if (lane + d < 32) {
                    b = axpy_(c, bp, b);
                    c = mul_(c, cp);
                }
            }
            const double c0 = shfl_idx(c, 0), b0 = shfl_idx(b, 0);
            if (lane < kNC) {
                Shared* const R = cluster.map_shared_rank(&S, lane);
                R->cb[w] = c0;
                R->bb[w] = b0;
            }
        }
        cluster.sync();
        double s2 = 0.0;
        if (sub == 0) {
            double uin = 0.0;
            for (int q = kWarps - 1; q > w; q--) uin = axpy_(S.cb[q], uin, S.bb[q]);
            {
                const double cp = shfl_down(c, 1), bp = shfl_down(b, 1);
                uin = lane == 31 ? uin : axpy_(cp, uin, bp);
            }
            for (int i = 0; i < m; i++) {
                const int q = i * kT + lane;
                const double u = fma(GG[q], uin, yl[q]);
                yl[q] = u;
                s2 = fma(u, u, s2);
            }
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) s2 += shfl_xor(s2, d);
            if (lane < kNC) cluster.map_shared_rank(&S, lane)->norm[w] = s2;
        }
        cluster.sync();
        s2 = 0.0;
#pragma unroll
        for (int q = 0; q < kWarps; q++) s2 += S.norm[q];
        const double nrm = sqrt(s2);  // normalise (tools.c:137-145)
        for (int i = sub; i < m; i += kSub) psi[i * kT + lane] = yl[i * kT + lane] / nrm;
        send_edges();
        cluster.sync();
        // ---- energy quotient (tridiag.c:172-238): the terms by all warps, each chunk's sum by its own
        for (int i = sub; i < m; i += kSub) {
            const int q = i * kT + lane;
            const double pm = i > 0 ? psi[q - kT] : lane == 0 ? S.left : psi[(m - 1) * kT + lane - 1];
            const double pn = i + 1 < m ? psi[q + kT] : lane == 31 ? S.right : psi[lane + 1];
            const double vm = i > 0 ? vq[q - kT] : vl, vn = i + 1 < m ? vq[q + kT] : vr;
            double kpsi, mpsi;
            quotient_terms(inv_dx2, pm, psi[q], pn, vm, vq[q], vn, i, m, kpsi, mpsi);
            yl[q] = kpsi;
            mq[q] = mpsi;
        }
        __syncthreads();
        double acc[2] = {0.0, 0.0};
        if (sub == 0) {
            for (int i = 0; i < m && (int64_t)t * m + i < n; i++) {
                const int q = i * kT + lane;
                acc[0] = fma(yl[q], mq[q], acc[0]);
                acc[1] = fma(mq[q], mq[q], acc[1]);
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
#pragma unroll
                for (int d = 16; d >= 1; d >>= 1) acc[k] += shfl_xor(acc[k], d);
                if (lane < kNC) cluster.map_shared_rank(&S, lane)->quot[w * 2 + k] = acc[k];
            }
        }
        cluster.sync();
#pragma unroll
        for (int k = 0; k < 2; k++) {
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < kWarps; q++) s += S.quot[q * 2 + k];
            acc[k] = s;
        }
        energy = acc[0] / acc[1];
        test = fabs(energy - e_old);
        e_old = energy;
        ++it;
        if (it >= G.max_iter) {
            status = MMA_ERR_GS_NOCONV;
            break;
        }
        if (!(test > G.CV)) break;
    }
    // final normalisation (tridiag.c:150)
    if (sub == 0) {
        double s2 = 0.0;
        for (int i = 0; i < m; i++) s2 = fma(psi[i * kT + lane], psi[i * kT + lane], s2);
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) s2 += shfl_xor(s2, d);
        if (lane < kNC) cluster.map_shared_rank(&S, lane)->norm[w] = s2;
    }
    cluster.sync();  // and no CTA leaves while another may still write to it
    double s2 = 0.0;
#pragma unroll
    for (int q = 0; q < kWarps; q++) s2 += S.norm[q];
    const double nrm = sqrt(s2);
    for (int i = sub; i < m; i += kSub) {
        const int64_t j = (int64_t)t * m + i;
        if (j < n) st2(G.psi0 + 2 * j, cd{psi[i * kT + lane] / nrm, 0.0});
    }
    if (threadIdx.x == 0 && rank == 0) {
        G.result[0] = energy;
        G.result[1] = (double)it;
        G.result[2] = (double)status;
        G.result[3] = test;
    }
}

}  // namespace

namespace {
cudaLaunchConfig_t config(int n_grids, int64_t m, cudaStream_t st, cudaLaunchAttribute* at)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(n_grids * kNC));
    cfg.blockDim = dim3(kT * kSub);
    cfg.dynamicSmemBytes = sizeof(double) * kVectors * (size_t)m * kT;
    cfg.stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = kNC;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}
}  // namespace

bool ground_state_fits(int n_grids, int64_t m, int sms)
{
    if (n_grids * 4 > sms) return false;
    // all clusters resident at once, two CTAs an SM where they are more than the SMs
    if (sizeof(double) * kVectors * (size_t)m * kT > (n_grids * kNC > sms ? 110 : 220) * (size_t)1024) return false;
    cudaLaunchAttribute at{};
    const cudaLaunchConfig_t cfg = config(n_grids, m, nullptr, &at);
    int active = 0;
    return allow_smem(ground_state_cluster_kernel) == cudaSuccess &&
           succeeded(cudaOccupancyMaxActiveClusters(&active, ground_state_cluster_kernel, &cfg)) && active > 0;
}

bool ground_state_cluster(const mma_tdse_grid* grids_dev, int n_grids, int64_t m, cudaStream_t st)
{
    cudaLaunchAttribute at{};
    const cudaLaunchConfig_t cfg = config(n_grids, m, st, &at);
    return succeeded(cudaLaunchKernelEx(&cfg, ground_state_cluster_kernel, grids_dev, (int)m));
}

}  // namespace mma
