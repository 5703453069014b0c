// Fused longwave forward kernel (one CTA per column) and its launcher; the per-column
// algorithm is in lw_column.cuh.
#include "lw_column.cuh"

namespace rrtmgp_b200 {
namespace {

using namespace fused;

// DENSE: tables with more than three minor intervals over some g-point (tau_abs).
template <int CL, bool DENSE, int THREADS = 512, int PER_SM = 1>
__global__ void __launch_bounds__(THREADS, PER_SM) lw_forward_kernel(const KdistView<float> k, const LwGridIo io)
{
    lw_forward_column<CL, true, DENSE>(CtaCtx{}, k, io);
}

// Few columns: one thread-block cluster of `parts` CTAs per column, each a share of its g-points
// (SplitCtx; xch: offset of its exchange buffer).
template <int CL, bool DENSE>
__global__ void __launch_bounds__(512) lw_forward_split_kernel(const KdistView<float> k, const LwGridIo io, int parts, int xch)
{
    lw_forward_column<CL, true, DENSE>(SplitCtx{parts, xch}, k, io);
}

// Columns of more than 16 chunks: one thread-block cluster of cs CTAs per column (ClusterCtx).
template <int CL, bool DENSE>
__global__ void __launch_bounds__(512) lw_forward_cluster_kernel(const KdistView<float> k, const LwGridIo io, int cs)
{
    lw_forward_column<CL, true, DENSE>(ClusterCtx<CL>{cs}, k, io);
    cooperative_groups::this_cluster().sync();   // no CTA leaves while another may store into its shared memory
}

// The instance for columns of NW chunks of 8 layers whose CTAs take smem bytes: register caps that let
// more CTAs share an SM, as the kernel waits on table loads (16 warps per SM at 128 registers).  At
// 80 registers (40 bytes of spill loads) an SM holds 24 warps; 9 and 10 chunks need none at 96.  Only
// where the CTAs fit and some SM gets more than one (crowded: more columns than SMs): 147 x 72 unsplit takes
// 54 us at 128 registers, 58 at 96.
template <int CL, bool DENSE>
auto pick_forward(int NW, size_t smem, bool crowded) -> void (*)(const KdistView<float>, const LwGridIo)
{
    if constexpr (CL == 8) {
        if (crowded && NW <= 8 && ctas_fit(3, smem)) return lw_forward_kernel<CL, DENSE, 256, 3>;
        if (crowded && NW > 8 && NW <= 10 && ctas_fit(2, smem)) return lw_forward_kernel<CL, DENSE, 320, 2>;
        if (crowded && NW > 10 && NW <= 12 && ctas_fit(2, smem)) return lw_forward_kernel<CL, DENSE, 384, 2>;
    }
    return lw_forward_kernel<CL, DENSE>;
}

// Shared-memory limits of the instances on the current device, set once.
template <int CL, bool DENSE>
int lw_forward_attributes()
{
    static PerDeviceOnce attr;
    return attr.run([] {
        for (int nw : {8, 10, 12, 16, 17}) {   // every instance
            const cudaError_t e = cudaFuncSetAttribute(pick_forward<CL, DENSE>(nw, 0, nw < 17),
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
            if (e != cudaSuccess) return e;
        }
        const cudaError_t e2 = cudaFuncSetAttribute(lw_forward_split_kernel<CL, DENSE>,
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e2 != cudaSuccess) return e2;
        return cudaFuncSetAttribute(lw_forward_cluster_kernel<CL, DENSE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    220 * 1024);
    }, "forward_lw attribute");
}

// Shared memory of one of the CS CTAs of a column (NWc chunks of CL layers each).
template <int CL>
size_t lw_forward_smem(const KdistView<float>& v, int NWc, int CS)
{
    return smem_layout(NWc * CL, v.ngas, v.nband, 1, CS * NWc, 2, CL, v.max_group_bands * (CL == 8 ? 2 : 1),
                       v.max_nscal, sizeof(LwRec), NWc).total;
}

// Columns that the device holds at once, one CTA each in chunks of CL layers; 0 when they do not fit.
template <int CL, bool DENSE>
int lw_columns_at_once(rrtmgp_b200_kdist k, int ncol, int nlay)
{
    const int NW = ceil_div(nlay, CL);
    const size_t smem = lw_forward_smem<CL>(k->v32, NW, 1);
    if (smem > 220 * 1024 || lw_forward_attributes<CL, DENSE>()) return 0;
    return resident(pick_forward<CL, DENSE>(NW, smem, ncol > k->nsm), k->nsm, NW * 32, smem, 1);
}

// Default chunk length.  8 and 16 layers hold different numbers of columns at once (72 layers: 296 and
// 444), and a wave of the latter takes 1.4 - 1.65 times one of the former, so the shorter time in whole
// waves is taken at 1.5 (us, 8 and 16 layers: 400 x 72 121 and 97, 520 x 72 130 and 184, 520 x 60 134
// and 99, 700 x 60 135 and 193, 400 x 112 177 and 199, 590 x 112 236 and 207; large grids 4096 x 91 1.12 and
// 1.26 ms, 8192 x 128 3.24 and 2.93 ms).  Grids of up to one column per SM, split or not, are faster with
// 8 up to 96 layers.  More than 128 layers need 16 to fit one CTA.
template <bool DENSE>
int lw_chunk(rrtmgp_b200_kdist k, int ncol, int nlay)
{
    if (nlay > 128) return 16;
    if (ncol > k->nsm) {
        const int n8 = lw_columns_at_once<8, DENSE>(k, ncol, nlay), n16 = lw_columns_at_once<16, DENSE>(k, ncol, nlay);
        if (n8 > 0 && n16 > 0) return 2 * ceil_div(ncol, n8) <= 3 * ceil_div(ncol, n16) ? 8 : 16;
    }
    return nlay <= 96 ? 8 : 16;
}

template <int CL, bool DENSE>
int launch_lw_forward(rrtmgp_b200_kdist k, rrtmgp_b200_cloud c, int ncol, int nlay, const float* play,
                      const float* plev, const float* tlay, const float* tlev, const float* tsfc, const float* col_dry,
                      const GasSet<float>& gs, const float* lwp, const float* iwp, const float* rel, const float* rei,
                      const float* emis, float* up, float* dn, float* net, float* hr, cudaStream_t stream)
{
    const KdistView<float>& v = k->v32;
    const int NW = (nlay + CL - 1) / CL;
    // more than 16 chunks: a cluster of CS CTAs of NWc warps per column
    const int CS = (NW + 15) / 16, NWc = (NW + CS - 1) / CS;
    RB_CHECK_ARG(CS <= 8, "forward_lw: nlay too large for the fused kernel (at most 128 chunks)");
    const size_t smem = lw_forward_smem<CL>(v, NWc, CS);
    if (smem > 220 * 1024) return fail(RRTMGP_B200_ERR_UNSUPPORTED, "forward_lw: shared memory need exceeds 220 KB");
    if (const int st = lw_forward_attributes<CL, DENSE>()) return st;
    CloudArgs ca{};
    if (c) {
        ca.L = CloudLut<float>{c->nband, c->nsize_liq, c->nsize_ice, float(c->radliq_lwr), float(c->liq_step),
                               float(c->radice_lwr), float(c->ice_step), c->lut32};
        ca.lwp = lwp; ca.iwp = iwp; ca.rel = rel; ca.rei = rei;
        ca.present = 1;
    }
    LwGridIo io{ncol, nlay, play, plev, tlay, tlev, tsfc, col_dry, emis, up, dn, net, hr, gs, ca};
    // the split's exchange buffer: 4 accumulators per thread
    const size_t xch = align16(smem), split_smem = xch + sizeof(double) * 4 * NW * 32;
    const auto whole = pick_forward<CL, DENSE>(NW, smem, ncol > k->nsm);
    const auto ask = [&](int s) {
        return s == 1 ? resident(whole, k->nsm, NW * 32, smem, 1)
                      : resident(lw_forward_split_kernel<CL, DENSE>, k->nsm, NW * 32, split_smem, s);
    };
    const int parts = CS > 1 || split_smem > 227 * 1024
                          ? 1 : group_parts(ncol, v.ngroups, residency()(whole, k->device, NW * 32, smem, ask));
    if (CS == 1 && parts == 1) {
        whole<<<ncol, NW * 32, smem, stream>>>(v, io);
        RB_LAUNCH("lw_forward_kernel");
        return RRTMGP_B200_OK;
    }
    cudaLaunchConfig_t cfg = {};
    const int cluster = CS == 1 ? parts : CS;
    cfg.gridDim = dim3(unsigned(ncol) * cluster);
    cfg.blockDim = dim3(NWc * 32);
    cfg.dynamicSmemBytes = CS == 1 ? split_smem : smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = unsigned(cluster);
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (CS == 1) {
        RB_CUDA(cudaLaunchKernelEx(&cfg, lw_forward_split_kernel<CL, DENSE>, v, io, parts, int(xch)),
                "lw_forward_split_kernel");
        return RRTMGP_B200_OK;
    }
    RB_CUDA(cudaLaunchKernelEx(&cfg, lw_forward_cluster_kernel<CL, DENSE>, v, io, CS), "lw_forward_cluster_kernel");
    return RRTMGP_B200_OK;
}

}  // namespace

int forward_lw_f32(rrtmgp_b200_kdist k, rrtmgp_b200_cloud c, int ncol, int nlay, const float* play,
                   const float* plev, const float* tlay, const float* tlev, const float* tsfc, const float* col_dry,
                   const rrtmgp_b200_gas_conc* gases, int ngases, const float* lwp, const float* iwp,
                   const float* rel, const float* rei, const float* sfc_emis, float* flux_up, float* flux_dn,
                   float* flux_net, float* heating_rate, int chunk, void* stream)
{
    RB_CHECK_ARG(k && k->info.is_longwave, "forward_lw: need a longwave k-distribution");
    if (const int dst = check_device(k->device, "forward_lw")) return dst;
    RB_CHECK_ARG(ncol > 0 && nlay > 1, "forward_lw: ncol > 0 and nlay > 1 required");
    RB_CHECK_ARG(play && plev && tlay && tlev && tsfc && sfc_emis && flux_up && flux_dn && flux_net && heating_rate,
                 "forward_lw: null array");
    RB_CHECK_ARG(!c || (lwp && iwp && rel && rei), "forward_lw: cloud arrays required with a cloud handle");
    RB_CHECK_ARG(!c || c->nband == k->info.nband, "forward_lw: cloud and gas band counts differ");
    const KdistView<float>& v = k->v32;
    if (!fused_layout_ok(v, false, 8))
        return fail(RRTMGP_B200_ERR_UNSUPPORTED, "forward_lw: k-distribution layout not supported by the fused kernel");
    GasSet<float> gs;
    int st = make_gas_set<float>(k, ncol, nlay, gases, ngases, gs);
    if (st) return st;
    cudaStream_t s = as_stream(stream);
    const bool dense = v.max_minor_per_g > 3;
#define RB_LW_FWD(CLv, D)                                                                                          \
    launch_lw_forward<CLv, D>(k, c, ncol, nlay, play, plev, tlay, tlev, tsfc, col_dry, gs, lwp, iwp, rel, rei, \
                              sfc_emis, flux_up, flux_dn, flux_net, heating_rate, s)
    if (chunk == 0) chunk = dense ? lw_chunk<true>(k, ncol, nlay) : lw_chunk<false>(k, ncol, nlay);
    if (chunk == 8) return dense ? RB_LW_FWD(8, true) : RB_LW_FWD(8, false);
    return dense ? RB_LW_FWD(16, true) : RB_LW_FWD(16, false);
#undef RB_LW_FWD
}

}  // namespace rrtmgp_b200

extern "C" int rrtmgp_b200_forward_lw_f32(rrtmgp_b200_kdist k, rrtmgp_b200_cloud c, int ncol, int nlay,
        const float* play, const float* plev, const float* tlay, const float* tlev, const float* tsfc,
        const float* col_dry, const rrtmgp_b200_gas_conc* gases, int ngases, const float* lwp, const float* iwp,
        const float* rel, const float* rei, const float* sfc_emis, float* flux_up, float* flux_dn, float* flux_net,
        float* heating_rate, int chunk, void* stream)
{
    return rrtmgp_b200::forward_lw_f32(k, c, ncol, nlay, play, plev, tlay, tlev, tsfc, col_dry, gases, ngases, lwp,
                                       iwp, rel, rei, sfc_emis, flux_up, flux_dn, flux_net, heating_rate, chunk, stream);
}
