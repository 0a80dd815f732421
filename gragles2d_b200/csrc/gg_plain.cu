// Plain form: FP64 kernels compiled without FMA contraction (--fmad=false),
// so every sum, product and quotient rounds exactly as the reference's
// host arithmetic does.
#include "gg_corrector.cuh"
#include "gg_dft.cuh"
#include "gg_kernels.cuh"
#include "gg_launch.cuh"
#include "gg_redist.cuh"
#include "gg_tangent.cuh"
#include "gg_warp.cuh"

namespace gg {

// Corrector of the plain form (LSbox::executeConvolution, src/box.cpp:428-531):
// the sectors come from k_sectors; each warp takes 8 x 4 tiles of the box and
// finds its pixels' nearest vertices as above; the segment, the weight and the
// blend are the reference's FP64 expressions.  Contours longer than kCorrPts
// are searched in FP64 from device memory.  Bound by instruction issue and by
// the FP64 divisions of the segment step; 5,000 grains 1.24 -> 0.64 ms with
// k_sectors (before: the sectors built inside, every vertex measured in FP64).
struct PlainCorrectorSmem {
    float2 sp[kCorrPts];
    float4 list[4][kTileList];
    double acc[kCorrPts];
    double cw[kMaxConstSectors];
    InterpSector is[kMaxInterpSectors];
    NbTable nbt;
    int16_t sid[kCorrPts];
};

__global__ void __launch_bounds__(128, 6) k_corrector(NetConst C, NetState* S) {
    const int g = blockIdx.x + 1;
    if (g > C.N || C.state[g] != G_EXISTS || C.regular[g] == 0 || S->loop == 0 || halted(S)) return;
    __shared__ __align__(16) PlainCorrectorSmem sm;
    const int64_t coff = S->coff_prev[g];
    const CPoint* P = S->contPrev + coff;
    const int size = S->cn_prev[g];
    if (size < 2) return;
    const Box ib = S->box_prev[g];
    const uint32_t* idl = S->idPrev + S->off_prev[g];
    const bool staged = size <= kCorrPts;
    const SectorPack* pk = reinterpret_cast<const SectorPack*>(C.secpack) + g;
    const int nconst = pk->nconst, ninterp = pk->ninterp;
    for (int c = threadIdx.x; c < nconst; c += blockDim.x) sm.cw[c] = pk->cw[c];
    for (int c = threadIdx.x; c < ninterp; c += blockDim.x) sm.is[c] = pk->is[c];
    const int16_t* tsid = C.segsec + coff;
    const double* tacc = C.segacc64 + coff;
    float span = 0.f;
    if (staged) {
        for (int k = threadIdx.x; k < size; k += blockDim.x)
            sm.sp[k] = make_float2((float)(P[k].x - ib.x0), (float)(P[k].y - ib.y0));
        for (int q = threadIdx.x; q < size - 1; q += blockDim.x) {
            sm.sid[q] = tsid[q];
            sm.acc[q] = tacc[q];
        }
        tsid = sm.sid;
        tacc = sm.acc;
    }
    build_nb_table(C, g, sm.nbt);
    __syncthreads();
    if (staged) span = staged_span(sm.sp, size, box_w(ib), box_h(ib));
    const Box bo = S->box_cur[g];
    const int x0 = ib.x0 < bo.x0 ? bo.x0 : ib.x0;
    const int y0 = ib.y0 < bo.y0 ? bo.y0 : ib.y0;
    const int x1 = ib.x1 > bo.x1 ? bo.x1 : ib.x1;
    const int y1 = ib.y1 > bo.y1 ? bo.y1 : ib.y1;
    if (x1 <= x0 || y1 <= y0) return;
    const int w = x1 - x0, hgt = y1 - y0;
    const double* in = phiA_of<double>(S) + S->off_cur[g];
    double* out = phiB_of<double>(S) + S->off_cur[g];
    const int wo = box_w(bo), real = size - 1;
    const double delta = C.delta;
    const bool forces = C.stored || C.magnetic;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int ntx = (w + 7) >> 3, ntiles = ntx * ((hgt + 3) >> 2);
    uint32_t st = 0;
    for (int t = warp; t < ntiles; t += nwarps) {
        const int tx = x0 + (t % ntx) * 8, ty = y0 + (t / ntx) * 4;
        const int j = tx + (lane & 7), i = ty + (lane >> 3);
        const bool inside = j < x1 && i < y1;
        const int k = (i - bo.y0) * wo + (j - bo.x0);
        double val = 0, conv = 0;
        if (inside) {
            val = in[k];
            conv = out[k];
        }
        const bool need = inside && val > -delta;
        double result = -delta;
        if (__any_sync(0xffffffffu, need)) {
            double lambda = 0.0;
            int segment = 0;
            if (staged) {
                const int nv = nearest_vertex_tile(sm.sp, P, real, tx, ty, j, i, ib.x0, ib.y0, span, need, sm.list[warp]);
                if (need && nv >= 0) segment = segment_of_vertex(P, size, (double)j, (double)i, nv, &lambda);
            } else if (need) {
                segment = project_to_boundary(P, size, (double)j, (double)i, &lambda);
            }
            if (need) {
                const double weight = segment_weight(C, sm.nbt, P, real, tsid[segment], tacc[segment], sm.cw, sm.is,
                                                     segment, lambda, idl, ib, i, j, &st);
                result = val + (conv - val) * weight * 1.0;
            }
        }
        if (inside) {
            if (forces) result = subtract_driving_forces<double>(C, sm.nbt, idl, ib, i, j, result, &st);
            out[k] = result;
        }
    }
    if (st) set_status(S, st);
}

__global__ void k_swap_phi(NetState* S) {
    void* t = S->phiA;
    S->phiA = S->phiB;
    S->phiB = t;
    t = S->dphiA;
    S->dphiA = S->dphiB;
    S->dphiB = t;
}

cudaError_t swap_phi(NetState* dS, cudaStream_t s) {
    k_swap_phi<<<1, 1, 0, s>>>(dS);
    return cudaGetLastError();
}

cudaError_t plain_resample(const NetConst& C, NetState* dS, double h_old, double hn, double delta_old,
                           cudaStream_t s) {
    if (C.N > 0) k_resample<double><<<C.N, 256, 0, s>>>(C, dS, h_old, hn, delta_old);
    return cudaGetLastError();
}

// The per-grain statistics of gg_read_grain_stats, gathered into one array.
__global__ void k_pack_stats(NetConst C, const NetState* S, gg_grain_stats* out) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (g > C.N) return;
    gg_grain_stats s;
    s.id = g;
    s.state = C.state[g];
    s.motion_regular = C.regular[g];
    s.intersects_boundary = C.inter_bnd[g];
    s.n_neighbours = C.nb_n[g];
    s.contour_points = S->cn_prev[g];
    const Box b = S->box_cur[g];
    s.box[0] = b.x0;
    s.box[1] = b.x1;
    s.box[2] = b.y0;
    s.box[3] = b.y1;
    s.area = C.volume[g];
    s.energy = C.energy[g];
    s.perimeter = C.perimeter[g];
    s.mean_da = C.meanda[g];
    out[g - 1] = s;
}

cudaError_t pack_stats(const NetConst& C, const NetState* dS, gg_grain_stats* out, cudaStream_t s) {
    if (C.N > 0) k_pack_stats<<<(C.N + 255) / 256, 256, 0, s>>>(C, dS, out);
    return cudaGetLastError();
}

cudaError_t finalize_only(const NetConst& C, NetState* dS, int rotate, cudaStream_t s) {
    k_finalize<<<1, 1024, 0, s>>>(C, dS, rotate);
    return cudaGetLastError();
}

cudaError_t neighbour_bins_count(const NetConst& C, NetState* dS, const NeighbourBins& B, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(B.count, 0, sizeof(int) * (size_t)B.nc * B.nc, s);
    if (e != cudaSuccess) return e;
    if (C.N > 0) k_bin_grains<<<(C.N + 255) / 256, 256, 0, s>>>(C, dS, B, 0);
    k_bin_scan<<<1, 1024, 0, s>>>(B);
    return cudaGetLastError();
}

cudaError_t find_neighbors_launch(const NetConst& C, NetState* dS, const NeighbourBins& B, cudaStream_t s) {
    if (C.N <= 0) return cudaSuccess;
    k_bin_grains<<<(C.N + 255) / 256, 256, 0, s>>>(C, dS, B, 1);
    k_find_neighbors<<<(C.N + kFindWarps - 1) / kFindWarps, 32 * kFindWarps, 0, s>>>(C, dS, B);
    return cudaGetLastError();
}

// Dynamic shared memory above the default limit (per device, before the first launch).
cudaError_t plain_prepare() {
    const auto allow = [](auto* kernel, size_t bytes) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    cudaError_t e = allow(k_conv_dft_s<0>, dft_smem(DftBin<0>::kHigh));
    if (e == cudaSuccess) e = allow(k_conv_dft_s<1>, dft_smem(DftBin<1>::kHigh));
    if (e == cudaSuccess) e = allow(k_conv_dft_s<2>, dft_smem(DftBin<2>::kHigh));
    if (e == cudaSuccess) e = allow(k_redistance<double, false>, redist_smem<double, false>());
    if (e == cudaSuccess) e = allow(k_redistance<double, true>, redist_smem<double, true>());
    if (e == cudaSuccess) e = allow(k_redistance_ts<false>, sizeof(RedistTangentCta<false>));
    if (e == cudaSuccess) e = allow(k_redistance_ts<true>, sizeof(RedistTangentCta<true>));
    return e;
}

// The distance field's convolution, with `tangents` that of its four tangent
// fields, and beside it with `sectors` the corrector's sectors.
cudaError_t launch_convolution_plain(const NetConst& C, NetState* dS, cudaStream_t s, const LaunchCfg& cfg,
                                     bool tangents, bool sectors) {
    const dim3 grid(C.N, tangents ? 1 + kNP : 1);
    cudaError_t e;
    if ((e = cudaEventRecord(cfg.ev[0], s)) != cudaSuccess) return e;
    for (int k = 0; k < 2; ++k)
        if ((e = cudaStreamWaitEvent(cfg.side[k], cfg.ev[0], 0)) != cudaSuccess) return e;
    k_conv_dft_s<2><<<grid, DftBin<2>::kThreads, dft_smem(DftBin<2>::kHigh), cfg.side[0]>>>(C, dS);
    k_conv_dft<<<C.N, 256, 0, cfg.side[0]>>>(C, dS, tangents ? kNP : 0);
    if (sectors) k_sectors<false, double><<<C.N, 32, 0, cfg.side[1]>>>(C, dS);
    k_conv_dft_s<1><<<grid, DftBin<1>::kThreads, dft_smem(DftBin<1>::kHigh), cfg.side[1]>>>(C, dS);
    k_conv_dft_s<0><<<grid, DftBin<0>::kThreads, dft_smem(DftBin<0>::kHigh), s>>>(C, dS);
    for (int k = 0; k < 2; ++k) {
        if ((e = cudaEventRecord(cfg.ev[1 + k], cfg.side[k])) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(s, cfg.ev[1 + k], 0)) != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

void launch_levelset_plain(const NetConst& C, NetState* dS, cudaStream_t s) {
    k_levelset_big<double><<<C.N, 32, 0, s>>>(C, dS);
    k_levelset_w<double><<<(C.N + kGrainsPerBlock - 1) / kGrainsPerBlock, 32 * kGrainsPerBlock, 0, s>>>(C, dS);
}

void launch_redistance_plain(const NetConst& C, NetState* dS, cudaStream_t s) {
    k_redistance<double, true><<<C.N, redist_threads<double, true>(), redist_smem<double, true>(), s>>>(C, dS);
    k_redistance<double, false><<<C.N, kRedistThreads, redist_smem<double, false>(), s>>>(C, dS);
}

void launch_redistance_tangent(const NetConst& C, NetState* dS, cudaStream_t s) {
    k_redistance_t<<<C.N, 64, 0, s>>>(C, dS);  // boxes that do not stage
    k_redistance_ts<true><<<C.N, kRedistTThreads, sizeof(RedistTangentCta<true>), s>>>(C, dS);
    k_redistance_ts<false><<<C.N, kRedistThreads, sizeof(RedistTangentCta<false>), s>>>(C, dS);
}

cudaError_t plain_init(const NetConst& C, NetState* dS, const int32_t* d_ids, cudaStream_t s) {
    if (C.N <= 0) return cudaSuccess;
    k_init_phi<double><<<C.N, 256, 0, s>>>(C, dS, d_ids);
    launch_redistance_plain(C, dS, s);
    k_swap_phi<<<1, 1, 0, s>>>(dS);
    k_init_contour_big<double><<<C.N, 32, 0, s>>>(C, dS);
    k_init_contour_w<double><<<(C.N + kGrainsPerBlock - 1) / kGrainsPerBlock, 32 * kGrainsPerBlock, 0, s>>>(C, dS);
    return cudaGetLastError();
}

cudaError_t plain_init_polygon(const NetConst& C, NetState* dS, cudaStream_t s) {
    if (C.N <= 0) return cudaSuccess;
    k_polygon_phi<double><<<C.N, 256, 0, s>>>(C, dS);
    return cudaGetLastError();
}

cudaError_t traffic_launch(const NetConst& C, NetState* dS, cudaStream_t s) {
    const int gt = 128;
    k_traffic<<<(C.N + gt - 1) / gt, gt, 0, s>>>(C, dS);
    return cudaGetLastError();
}

cudaError_t plain_stage_kernel(const NetConst& C, NetState* dS, int which, cudaStream_t s, const LaunchCfg& cfg) {
    const int wblocks = (C.N + kGrainsPerBlock - 1) / kGrainsPerBlock;
    switch (which) {
        case 0: return launch_convolution_plain(C, dS, s, cfg, false, false);
        case 1:
            if (!C.isotropic) {
                k_sectors<false, double><<<C.N, 32, 0, s>>>(C, dS);
                k_corrector<<<C.N, 128, 0, s>>>(C, dS);
            }
            break;
        case 2: k_second_order_w<<<wblocks, 32 * kGrainsPerBlock, 0, s>>>(C, dS); break;
        case 3: k_compare<double><<<C.N, cfg.compare_threads, 0, s>>>(C, dS); break;
        case 4: launch_levelset_plain(C, dS, s); break;
        case 5: k_alloc<<<1, 1024, 0, s>>>(C, dS, 2); break;
        case 6: k_neighbours_w<double><<<wblocks, 32 * kGrainsPerBlock, 0, s>>>(C, dS, reinterpret_cast<PointInfo*>(C.ptinfo)); break;
        case 7: launch_redistance_plain(C, dS, s); break;
        default: k_finalize<<<1, 1024, 0, s>>>(C, dS, 1); break;
    }
    return cudaGetLastError();
}

cudaError_t plain_stages(const NetConst& C, NetState* dS, int stages, cudaStream_t s, const LaunchCfg& cfg) {
    if (C.N <= 0) return cudaSuccess;
    const int wblocks = (C.N + kGrainsPerBlock - 1) / kGrainsPerBlock;
    // tangent mode (C.dvol set): the tangent kernels of gg_tangent.cuh follow
    // their stages; the corrector's tangent reads the uncorrected convolution,
    // so it runs first
    const bool tan = C.dvol != nullptr;
    if (stages & ST_CONV) {
        cudaError_t ec = launch_convolution_plain(C, dS, s, cfg, tan, !C.isotropic);
        if (ec != cudaSuccess) return ec;
        if (!C.isotropic) {
            if (tan) k_corrector_t<<<C.N, 128, 0, s>>>(C, dS);
            k_corrector<<<C.N, 128, 0, s>>>(C, dS);
        }
    }
    if (stages & ST_SECOND) k_second_order_w<<<wblocks, 32 * kGrainsPerBlock, 0, s>>>(C, dS);
    if (stages & ST_COMPARE) {
        k_compare<double><<<C.N, cfg.compare_threads, 0, s>>>(C, dS);
        if (tan) k_compare_t<<<C.N, 256, 0, s>>>(C, dS);
    }
    if (stages & ST_LEVELSET) {
        launch_levelset_plain(C, dS, s);
        if (tan) k_area_t<<<(C.N + 3) / 4, 128, 0, s>>>(C, dS);  // warp per grain
    }
    if (stages & ST_REDIST) {
        k_alloc<<<1, 1024, 0, s>>>(C, dS, 2);
        k_neighbours_w<double><<<wblocks, 32 * kGrainsPerBlock, 0, s>>>(C, dS, reinterpret_cast<PointInfo*>(C.ptinfo));
        if (tan)
            launch_redistance_tangent(C, dS, s);
        else
            launch_redistance_plain(C, dS, s);
        k_finalize<<<1, 1024, 0, s>>>(C, dS, 1);
    }
    return cudaGetLastError();
}

}  // namespace gg
