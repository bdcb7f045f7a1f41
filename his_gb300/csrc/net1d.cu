// Launchers of the 1-D network kernels (float64, built with -fmad=false); float32
// engines run the production form's network (net1d_f32.cu).
#include "his_internal.h"
#include "net1d_kernels.cuh"

namespace his {

// n_sub substeps of dt/n_sub each for every member; forcing: dt, n_sub, then per member, per
// substep (inflow, stage); vols: 3 per member.
// ledger (optional): 8 x members float64 ledger; the substeps' boundary volumes and
// clip are added into its 1-D rows.
__global__ void __launch_bounds__(NET64_THREADS, 1) net_step_kernel(const Net* __restrict__ nets, Consts c,
                                const double* __restrict__ forcing, double* __restrict__ vols,
                                double* __restrict__ ledger) {
    extern __shared__ double sm[];
    __shared__ double v[3];
    const int n_sub = (int)forcing[1];
    net_substeps_dev(nets[blockIdx.x], c, forcing[0], n_sub, forcing + 2 + (size_t)blockIdx.x * n_sub * 2,
                     (vols || ledger) ? v : nullptr, sm);
    if (threadIdx.x == 0) {
        if (vols)
            for (int j = 0; j < 3; ++j) vols[blockIdx.x * 3 + j] = v[j];
        if (ledger) {
            const size_t B = gridDim.x;
            ledger[LG_BND1_IN * B + blockIdx.x] += v[0];
            ledger[LG_BND1_OUT * B + blockIdx.x] += v[1];
            ledger[LG_CLIP1 * B + blockIdx.x] += v[2];
        }
    }
}

// 1-D CFL rate over wet interior cells, the any-wet flag and the channel volume.
// out: 3 per member (rate, any_wet, volume).
__global__ void __launch_bounds__(NET64_THREADS) net_reduce_kernel(const Net* __restrict__ nets, Consts c,
                                                                   double* __restrict__ out,
                                                                   double* __restrict__ rate_wet) {
    __shared__ double s_rate[NET64_THREADS / 32], red[NET64_THREADS / 32];
    const Net& N = nets[blockIdx.x];
    double rate = -1.0, vol[1] = {0.0};
    for (int i = threadIdx.x; i < N.n_cells; i += blockDim.x) {
        if (N.kind[i] > 1) continue;
        const double A = N.A[i];
        vol[0] = fma(A, N.dx[i], vol[0]);
        const double r = cell_rate_1d(N, c, i, cell_depth(N, i, A), A, N.Q[i]);
        rate = r > rate ? r : rate;
    }
    for (int o = 16; o > 0; o >>= 1) rate = f64_max(rate, __shfl_xor_sync(0xffffffffu, rate, o));
    if ((threadIdx.x & 31) == 0) s_rate[threadIdx.x >> 5] = rate;
    block_sum<1>(vol, red);
    if (threadIdx.x == 0) {
        for (int k = 1; k < NET64_THREADS / 32; ++k) rate = f64_max(rate, s_rate[k]);
        const bool wet = f64_plus(rate);
        const double r = wet ? rate : 0.0, w = wet ? 1.0 : 0.0;
        out[blockIdx.x * 3 + 0] = r;
        out[blockIdx.x * 3 + 1] = w;
        out[blockIdx.x * 3 + 2] = vol[0];
        if (rate_wet) {
            rate_wet[blockIdx.x * 2 + 0] = r;
            rate_wet[blockIdx.x * 2 + 1] = w;
        }
    }
}

// Engine form: each member's dt, substep count and substep forcing come from the
// device (written by the engine's pre kernel); members not stepping are skipped.
__global__ void __launch_bounds__(NET64_THREADS, 1) net_engine_kernel(const Net* __restrict__ nets, Consts c, const EngMember* __restrict__ em,
                                  const StepParams* __restrict__ params, const double* __restrict__ netf, int max_sub,
                                  double* __restrict__ vol1d, int m0) {
    extern __shared__ double sm[];
    const int m = m0 + blockIdx.x;
    if (!params[m].active) return;
    const EngMember& E = em[m];
    const StepParams& P = params[m];
    net_substeps_dev(nets[m], c, E.dt, E.n_sub, netf + (size_t)m * max_sub * 2, vol1d + m * 3, sm, P.snap_eta,
                     P.snap_q, P.snap_ledger ? P.snap_ledger + L_V1D : nullptr);
}

int net_engine_prepare(his_engine* e) {
    if (e->grid->prec == HIS_PREC_F32) return net_engine_prepare_f32(e);
    if (e->net && e->net->smem > 48 * 1024)
        HIS_CK(cudaFuncSetAttribute(net_engine_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)e->net->smem));
    return HIS_OK;
}

int net_engine_launch(his_engine* e, cudaStream_t s, int m0, int count) {
    if (e->grid->prec == HIS_PREC_F32) return net_engine_launch_f32(e, s, m0, count);
    his_net* n = e->net;
    net_engine_kernel<<<count, NET64_THREADS, n->smem, s>>>(n->d_nets, n->c, e->d_em, e->grid->d_params, e->d_netf, e->max_sub,
                                                  e->d_vol1d, m0);
    HIS_CK(cudaGetLastError());
    return HIS_OK;
}

int net_step_launch(his_net* n, cudaStream_t s, double* vols, double* ledger) {
    if (n->smem > 48 * 1024)
        HIS_CK(cudaFuncSetAttribute(net_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n->smem));
    net_step_kernel<<<n->n, NET64_THREADS, n->smem, s>>>(n->d_nets, n->c, n->d_forcing,
                                               vols ? vols : (ledger ? nullptr : n->d_out), ledger);
    HIS_CK(cudaGetLastError());
    return HIS_OK;
}

int net_reduce_launch(his_net* n, cudaStream_t s, double* rate_wet) {
    net_reduce_kernel<<<n->n, NET64_THREADS, 0, s>>>(n->d_nets, n->c, n->d_out, rate_wet);
    HIS_CK(cudaGetLastError());
    return HIS_OK;
}

}  // namespace his
