// mpc_shapes.cuh -- per-grid-shape launch configuration of the pencil and plane sweeps.
//
// A shape variant fixes the device layout and both sweeps' launch shapes:
//   pencil tile  of the passes to and from real space: P = TP / Nt pencils, P * Nt / CH threads per
//                CTA (TP = 16384, CH = 32: one 512-thread CTA per SM; TP = 8192: two 256-thread CTAs
//                per SM; TP = 16384, CH = 16: one 1024-thread CTA per SM); the split step has its own
//                tile (step_kernel, mpc_step.cuh), the same for every variant of a grid;
//   SLO          slots interleaved in the layout (default 2 when P = 8, so t-rows are 128 B);
//   LD           no longer selects anything (every split-step tile is staged, mpc_step.cuh);
//   PMB          PL = 2: resident strip CTAs per SM the strip kernels are compiled for (0: 512 / PT,
//                at 128 registers; more CTAs hide more load latency at fewer registers each);
//   PL           plane passes: 1, one cluster kernel per sweep (plane_kernel); 2, the y part on
//                column strips and the x part on row strips, two kernels over HBM without
//                clusters (plane_y_kernel, plane_x_kernel), one more pass over HBM but every SM
//                busy and no cluster barrier; 3, as 2 with the y part staged by TMA bulk tensor
//                copies (plane_y_tma_kernel: persistent 256-thread CTAs, 3 unit buffers each);
//                4, the x part also by bulk copies, a warp per 4 KB of rows (plane_x_warp_kernel);
//                5, one pass with whole planes in shared memory (plane_smem_kernel, 64 x 64);
//   plane unit   PT threads per CTA and 512 / PT CTAs per SM, each CTA holding a
//                PLB = 128 KB * PT / 512 share of the unit; PL = 1: SLO == 2, the two interleaved
//                omega-planes split over CL CTAs; SLO == 1, planes larger than PLB split over
//                CL CTAs, smaller planes batched PB per CTA; PL = 2: strips of PLB bytes.
// Several variants of one grid may be compiled in; they differ only in speed.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <mutex>

#include "mpc_kernels.cuh"
#include "mpc_step.cuh"

namespace mpc {

// Launch of a sweep kernel, with `overlap` one that may start while the kernel before it drains (pdl_wait,
// mpc_tma.cuh; without, the wait returns at once), in clusters of CL CTAs.
template <class... KArgs, class... Args>
inline cudaError_t launch_sweep(void (*k)(KArgs...), int grid, int threads, int smem, cudaStream_t st, int CL, int overlap, const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (overlap) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (CL > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = CL;
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, k, args...);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link to libcuda)
inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    });
    return fn;
}

// The field (complex64, slot layout SLO = 1 in blocks of YB rows) as a FLOAT32 tensor of (2 Nx floats,
// YB rows, Ny / YB blocks, Nt slots), with boxes of box_x floats by whole columns.
inline cudaError_t field_tensor_map(CUtensorMap* m, const void* field, int Nx, int Ny, int Nt, int YB, int box_x) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return cudaErrorNotSupported;
    const cuuint64_t row = (cuuint64_t)Nx * 8, blk = row * YB;
    const cuuint64_t dims[4] = {(cuuint64_t)(2 * Nx), (cuuint64_t)YB, (cuuint64_t)(Ny / YB), (cuuint64_t)Nt};
    const cuuint64_t strides[3] = {row, blk * Nt, blk};
    const cuuint32_t box[4] = {(cuuint32_t)box_x, (cuuint32_t)YB, (cuuint32_t)(Ny / YB), 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(field), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// The same field as (2 RB floats of a row block's pencils, Nt / LL, LL, row blocks), with boxes of a warp's
// block of a split-step tile: P pencils by NB butterflies of LL positions (mpc_step.cuh).  The L2
// promotion (none, 64, 128 bytes) makes no difference.
inline cudaError_t pencil_tensor_map(CUtensorMap* m, const void* field, long NP, int Nt, int RB, int LL, int P, int NB) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return cudaErrorNotSupported;
    const cuuint64_t row = (cuuint64_t)RB * 8;
    const cuuint64_t dims[4] = {(cuuint64_t)(2 * RB), (cuuint64_t)(Nt / LL), (cuuint64_t)LL, (cuuint64_t)(NP / RB)};
    const cuuint64_t strides[3] = {row * LL, row, row * Nt};
    const cuuint32_t box[4] = {(cuuint32_t)(2 * P), (cuuint32_t)NB, (cuuint32_t)LL, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(field), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Resident-CTA grids of the persistent kernels on the context's device.  They and the kernel attributes are
// set for every context: the attributes belong to the current CUDA context (a device reset drops them, a
// second context has its own), the grids to a device's SM count.
struct LaunchGrids {
    int step = 0;                   // split step and diagnostics
    int strip_y = 0, strip_x = 0;   // strip kernels (PL = 2, 3), strip_y also plane_smem_kernel (PL = 5)
    int tma_y = 0, tma_x = 0;       // TMA y pass (PL = 3, 4), warp-per-unit x pass (PL = 4)
};

struct ShapeOps {
    int Nx, Ny, Nt, P, SLO, CL, PB, PT, CH, LD, PL;
    int lrb;   // log2 of the pencils of a row block of the layout (Nx Ny: whole planes)
    int step_tiles;   // tiles of the split step and the diagnostics
    int pencil_smem, plane_smem;
    cudaError_t (*setup)(LaunchGrids*);   // kernel attributes in the current context; grids for its device
    cudaError_t (*pencil)(int mode, const PencilArgs&, int grid, const LaunchGrids&, cudaStream_t);
    cudaError_t (*plane)(const PlaneArgs&, int nclusters, const LaunchGrids&, cudaStream_t);
    int (*max_clusters)(const LaunchGrids&);
    int (*pencil_blocks_per_sm)();   // resident pencil CTAs per SM (entry and exit modes)
};

template <int NX, int NY, int NT, int SLO_ = 0, int PT = kThreads, int TP = kTilePoints, int CH = 32, int LD = 1,
          int PL = 1, int PMB = 0>
struct Shape {
    static constexpr int P = TP / NT;
    static constexpr int SLO = SLO_ > 0 ? SLO_ : ((P < 16) ? 16 / P : 1);
    static constexpr long PLANE_B = (long)NX * NY * 8;
    static constexpr long PLB = 131072L * PT / kThreads;
    static constexpr int CL = PL >= 2 ? 1
                              : (SLO == 2) ? (int)(PLANE_B * 2 / PLB) : (PLANE_B > PLB ? (int)(PLANE_B / PLB) : 1);
    static constexpr int PB = PL >= 2 ? 1
                              : (SLO == 2) ? 2 : (PLANE_B > PLB ? 1 : ((PLB / PLANE_B) < NT ? (int)(PLB / PLANE_B) : NT));
    // PL = 2: column strips of CXS columns and row strips of RYS rows, PLB bytes each
    static constexpr int CXS = (int)(PLB / (NY * 8L)), RYS = (int)(PLB / (NX * 8L));
    static_assert(PL == 1 || (PL >= 2 && PL <= 5 && SLO == 1 && CXS >= 2 && CXS <= NX && RYS >= 1 && RYS <= NY),
                  "two-pass planes: SLO 1, strips within the plane");
    // PL = 3: the TMA-staged y pass on 16-column strips (128 B box rows), 256 threads, 3 buffers
    static constexpr int TCX = 16, TTH = 256, TNB = 3;
    static constexpr bool Y512 = PL == 4 && NY == 512;   // columns of 512 have a y pass of their own
    static_assert(PL < 3 || PL == 5 || NX % TCX == 0 && (NY <= 256 || Y512), "TMA boxes: 16 columns, at most 256 rows");
    // PL = 4: the x pass, XNW warps per CTA with XNB buffers each (plane_x_warp_kernel)
    static constexpr int SNW = 4, SMB = 4;   // PL = 5: warps per CTA and resident CTAs (plane_smem_kernel)
    static_assert(PL != 5 || (NX == 64 && NY == 64), "whole planes in shared memory");
    // layout: blocks of 16 rows for the large planes of PL = 4 (the other plane passes take whole
    // planes).  The split-step sweep, whole planes against 32, 16, 8, 4 rows: 256x256x2048 1.358 ms
    // against 1.261, 1.259, 1.260, 1.258; 512x512x1024 2.516 against 2.458, 2.454, 2.450, 2.450; the
    // plane sweep is the same for all.  Smaller planes fit the address translation caches as they are
    // (128x128x1024 gained nothing).
    static constexpr int YB = PL == 4 && (long)NX * NY >= 65536 ? 16 : NY;
    static_assert((PL != 3 && PL != 4) || NY > 128 || YB == NY, "plane_y_tma_kernel stores columns of up to 128 into whole planes");
    static constexpr int log2i(int n) { return n <= 1 ? 0 : 1 + log2i(n / 2); }
    static constexpr int LRB = log2i(YB * NX);
    static constexpr int XNW = 12, XNB = NX == 512 ? 4 : 3;
    static_assert(SLO == 1 || SLO == 2, "slot interleave");
    static_assert(PT == 128 || PT == 256 || PT == 512, "plane threads");
    static_assert(P >= 4 && P <= NX * NY, "pencil tile must fit the grid");
    static_assert(CL >= 1 && CL <= 16 && NY % CL == 0 && NX % CL == 0, "cluster split");
    using PC = PencilCfg<NT, P, SLO, CH>;
    using LC = PlaneCfg<NX, NY, CL, PB, SLO>;
    // Points of a split-step tile (mpc_step.cuh).  Nt <= 1024: 4096, two CTAs of 256 threads per SM, so that
    // one computes while the other waits at a barrier (8192 against 4096: 512x512x1024 2.264 against 2.155
    // ms, 128x128x1024 0.1578 against 0.1486, 256x256x512 0.2815 against 0.2735, 64x64x512 27.3 against
    // 26.8 us; 2048 at Nt = 512: 0.303 ms, 28.9 us).  Nt = 2048: 8192, whose 4 pencils make rows of 32 bytes.
    // Grids of fewer than 128 such tiles leave SMs idle: down to 1024 points, at least 8 pencils
    // (16x16x64 14.0 -> 10.0 us, 32x32x256 14.7 -> 11.6 us).
    static constexpr int step_tile(long n, int tp) { return n / tp >= 128 || tp <= 1024 || tp / 2 < 8 * NT ? tp : step_tile(n, tp / 2); }
    static constexpr int STP = step_tile((long)NX * NY * NT, NT <= 1024 ? 4096 : 8192);
    using SC = StepCfg<NT, STP>;
    static_assert((long)NX * NY % SC::P == 0, "whole split-step tiles");
    static constexpr int TH = PC::TH;

    static cudaError_t setup(LaunchGrids* grids) {
        cudaError_t e;
#define MPC_SET_SMEM(K, B)                                                                       \
    e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, B);                   \
    if (e != cudaSuccess) return e;
        MPC_SET_SMEM((pencil_kernel<NT, P, SLO, PM_ENTRY_C128, CH>), PC::SMEM);
        MPC_SET_SMEM((pencil_kernel<NT, P, SLO, PM_ENTRY_C64, CH>), PC::SMEM);
        MPC_SET_SMEM((step_kernel<NT, STP, SLO, LRB, true, true>), SC::SMEM);
        MPC_SET_SMEM((step_kernel<NT, STP, SLO, LRB, true, false>), SC::SMEM);
        MPC_SET_SMEM((step_kernel<NT, STP, SLO, LRB, false, true>), SC::SMEM);
        MPC_SET_SMEM((step_kernel<NT, STP, SLO, LRB, false, false>), SC::SMEM);
        {
            int dev = 0, nsm = 0, b = 0;
            if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
            if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
            if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, step_kernel<NT, STP, SLO, LRB, true, true>, SC::TH, SC::SMEM)) !=
                cudaSuccess)
                return e;
            if (b <= 0) return cudaErrorInvalidConfiguration;
            grids->step = b * nsm;
        }
        MPC_SET_SMEM((pencil_kernel<NT, P, SLO, PM_EXIT_C128, CH>), PC::SMEM);
        MPC_SET_SMEM((pencil_kernel<NT, P, SLO, PM_EXIT_C64, CH>), PC::SMEM);
        MPC_SET_SMEM((diag_kernel<NT, STP, SLO, LRB>), SC::DIAG_SMEM);
        MPC_SET_SMEM((pencil_kernel<NT, P, SLO, PM_IONIZ, CH>), PC::SMEM);
        if constexpr (PL == 5) {
            MPC_SET_SMEM((plane_smem_kernel<SNW, SMB>), PlaneS::SMEM);
            int dev = 0, nsm = 0, b = 0;
            if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
            if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, plane_smem_kernel<SNW, SMB>, SNW * 32, PlaneS::SMEM);
            if (e != cudaSuccess) return e;
            if (b <= 0) return cudaErrorInvalidConfiguration;
            grids->strip_y = b * nsm < NT ? b * nsm : NT;
            return cudaSuccess;
        } else if constexpr (PL >= 2) {
            int dev = 0, nsm = 0;
            if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
            if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
            if constexpr (PL == 4) {
                MPC_SET_SMEM((plane_x_warp_kernel<NX, YB, XNW, XNB>), XWarp<NX>::SMEM(XNW, XNB));
                grids->tma_x = nsm;
            }
            if constexpr (PL >= 3) {
                if (!tensor_map_encoder()) return cudaErrorNotSupported;
                int bt = 0;
                if constexpr (Y512) {
                    MPC_SET_SMEM((plane_y512_tma_kernel<NX>), StripY512::SMEM);
                    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bt, plane_y512_tma_kernel<NX>, StripY512::NTHR, StripY512::SMEM);
                } else {
                    MPC_SET_SMEM((plane_y_tma_kernel<NX, NY, TCX, TTH, TNB>), (StripYTmaCfg<NX, NY, TCX>::SMEM(TNB)));
                    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bt, plane_y_tma_kernel<NX, NY, TCX, TTH, TNB>, TTH,
                                                                      StripYTmaCfg<NX, NY, TCX>::SMEM(TNB));
                }
                if (e != cudaSuccess) return e;
                if (bt <= 0) return cudaErrorInvalidConfiguration;
                grids->tma_y = bt * nsm < NT * (NX / TCX) ? bt * nsm : NT * (NX / TCX);
            }
            MPC_SET_SMEM((plane_y_kernel<NX, NY, CXS, PT, PMB>), (StripYCfg<NX, NY, CXS>::SMEM));
            MPC_SET_SMEM((plane_x_kernel<NX, NY, RYS, PT, PMB>), (StripXCfg<NX, NY, RYS>::SMEM));
            int by = 0, bx = 0;
            if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&by, plane_y_kernel<NX, NY, CXS, PT, PMB>, PT,
                                                                   StripYCfg<NX, NY, CXS>::SMEM)) != cudaSuccess)
                return e;
            if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bx, plane_x_kernel<NX, NY, RYS, PT, PMB>, PT,
                                                                   StripXCfg<NX, NY, RYS>::SMEM)) != cudaSuccess)
                return e;
            grids->strip_y = by * nsm < NT * (NX / CXS) ? by * nsm : NT * (NX / CXS);
            grids->strip_x = bx * nsm < NT * (NY / RYS) ? bx * nsm : NT * (NY / RYS);
            return (by > 0 && bx > 0) ? cudaSuccess : cudaErrorInvalidConfiguration;
        } else {
            MPC_SET_SMEM((plane_kernel<NX, NY, CL, PB, SLO, PT>), LC::SMEM);
            if (CL > 8) {
                e = cudaFuncSetAttribute(plane_kernel<NX, NY, CL, PB, SLO, PT>,
                                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
                if (e != cudaSuccess) return e;
            }
            return cudaSuccess;
        }
#undef MPC_SET_SMEM
    }

    static cudaError_t pencil(int mode, const PencilArgs& a, int grid, const LaunchGrids& grids, cudaStream_t st) {
        switch (mode) {
            case PM_ENTRY_C128: pencil_kernel<NT, P, SLO, PM_ENTRY_C128, CH><<<grid, TH, PC::SMEM, st>>>(a); break;
            case PM_ENTRY_C64: pencil_kernel<NT, P, SLO, PM_ENTRY_C64, CH><<<grid, TH, PC::SMEM, st>>>(a); break;
            case PM_STEP: return step(a, grids.step, st);
            case PM_EXIT_C128: pencil_kernel<NT, P, SLO, PM_EXIT_C128, CH><<<grid, TH, PC::SMEM, st>>>(a); break;
            case PM_EXIT_C64: pencil_kernel<NT, P, SLO, PM_EXIT_C64, CH><<<grid, TH, PC::SMEM, st>>>(a); break;
            case PM_DIAG: return diag(a, grids.step, st);
            case PM_IONIZ: pencil_kernel<NT, P, SLO, PM_IONIZ, CH><<<grid, TH, PC::SMEM, st>>>(a); break;
            default: return cudaErrorInvalidValue;
        }
        return cudaGetLastError();
    }

    // the split-step sweep: persistent CTAs over tiles of STP points
    static cudaError_t step(const PencilArgs& args, int step_grid, cudaStream_t st) {
        PencilArgs a = args;
        a.ntiles = NX * NY / SC::P;
        const int g = step_grid < a.ntiles ? step_grid : a.ntiles;
        const bool sst = a.nl.sst_c != 0.0f;
        CUtensorMap tin{}, tout{};
        if constexpr (SLO == 1) {
            cudaError_t e;
            if ((e = pencil_tensor_map(&tin, a.in, (long)NX * NY, NT, YB * NX, SC::LL, SC::P, SC::NB)) != cudaSuccess) return e;
            if ((e = pencil_tensor_map(&tout, a.out, (long)NX * NY, NT, YB * NX, SC::LL, SC::P, SC::NB)) != cudaSuccess) return e;
        }
        if (sst && a.nl.plasma) return launch_sweep(step_kernel<NT, STP, SLO, LRB, true, true>, g, SC::TH, SC::SMEM, st, 1, 1, tin, tout, a);
        if (sst) return launch_sweep(step_kernel<NT, STP, SLO, LRB, true, false>, g, SC::TH, SC::SMEM, st, 1, 1, tin, tout, a);
        if (a.nl.plasma) return launch_sweep(step_kernel<NT, STP, SLO, LRB, false, true>, g, SC::TH, SC::SMEM, st, 1, 1, tin, tout, a);
        return launch_sweep(step_kernel<NT, STP, SLO, LRB, false, false>, g, SC::TH, SC::SMEM, st, 1, 1, tin, tout, a);
    }

    static cudaError_t diag(const PencilArgs& args, int step_grid, cudaStream_t st) {
        PencilArgs a = args;
        a.ntiles = NX * NY / SC::P;
        CUtensorMap tin{};
        if constexpr (SLO == 1) {
            const cudaError_t e = pencil_tensor_map(&tin, a.in, (long)NX * NY, NT, YB * NX, SC::LL, SC::P, SC::NB);
            if (e != cudaSuccess) return e;
        }
        diag_kernel<NT, STP, SLO, LRB><<<step_grid < a.ntiles ? step_grid : a.ntiles, SC::TH, SC::DIAG_SMEM, st>>>(tin, a);
        return cudaGetLastError();
    }

    // the TMA-staged y pass from `in` to `out` (tensor maps encoded per launch: a few host
    // microseconds, no device work)
    static cudaError_t plane_y_tma(const PlaneArgs& a, int second, int tma_grid_y, cudaStream_t st) {
        CUtensorMap tin, tout;
        cudaError_t e;
        if ((e = field_tensor_map(&tin, a.in, NX, NY, NT, YB, 2 * TCX)) != cudaSuccess) return e;
        if ((e = field_tensor_map(&tout, a.out, NX, NY, NT, YB, 2 * TCX)) != cudaSuccess) return e;
        if constexpr (Y512)
            return launch_sweep(plane_y512_tma_kernel<NX>, tma_grid_y, StripY512::NTHR, StripY512::SMEM, st, 1, a.overlap, tin, tout, a, second,
                                a.err);
        else
            return launch_sweep(plane_y_tma_kernel<NX, NY, TCX, TTH, TNB>, tma_grid_y, TTH, StripYTmaCfg<NX, NY, TCX>::SMEM(TNB), st, 1,
                                a.overlap, tin, tout, a, second, a.err);
    }

    // the x pass of PL = 4, in place on a.out
    static cudaError_t plane_x_warp(const PlaneArgs& a, int tma_grid_x, cudaStream_t st) {
        return launch_sweep(plane_x_warp_kernel<NX, YB, XNW, XNB>, tma_grid_x, XNW * 32, XWarp<NX>::SMEM(XNW, XNB), st, 1, a.overlap, a, a.err);
    }

    // the plain strip passes (PL = 2, 3)
    static cudaError_t plane_y(const PlaneArgs& a, int second, int strip_grid_y, cudaStream_t st) {
        return launch_sweep(plane_y_kernel<NX, NY, CXS, PT, PMB>, strip_grid_y, PT, StripYCfg<NX, NY, CXS>::SMEM, st, 1, a.overlap, a, second);
    }
    static cudaError_t plane_x(const PlaneArgs& a, int strip_grid_x, cudaStream_t st) {
        return launch_sweep(plane_x_kernel<NX, NY, RYS, PT, PMB>, strip_grid_x, PT, StripXCfg<NX, NY, RYS>::SMEM, st, 1, a.overlap, a);
    }

    static cudaError_t plane(const PlaneArgs& a, int nclusters, const LaunchGrids& grids, cudaStream_t st) {
        if constexpr (PL == 5) {
            return launch_sweep(plane_smem_kernel<SNW, SMB>, grids.strip_y, SNW * 32, PlaneS::SMEM, st, 1, a.overlap, a, a.err);
        } else if constexpr (PL == 4) {
            PlaneArgs b = a;
            b.in = a.out;   // the passes after the first run in place
            b.overlap = 1;
            cudaError_t e;
            if ((e = plane_y_tma(a, 0, grids.tma_y, st)) != cudaSuccess) return e;
            if ((e = plane_x_warp(b, grids.tma_x, st)) != cudaSuccess) return e;
            if (a.lens) return plane_y_tma(b, 1, grids.tma_y, st);
            return cudaSuccess;
        } else if constexpr (PL == 3) {
            PlaneArgs b = a;
            b.in = a.out;   // the passes after the first run in place
            b.overlap = 1;
            cudaError_t e;
            if ((e = plane_y_tma(a, 0, grids.tma_y, st)) != cudaSuccess) return e;
            if ((e = plane_x(b, grids.strip_x, st)) != cudaSuccess) return e;
            if (a.lens) return plane_y_tma(b, 1, grids.tma_y, st);
            return cudaSuccess;
        } else if constexpr (PL == 2) {
            PlaneArgs b = a;
            b.in = a.out;   // the passes after the first run in place
            b.overlap = 1;
            cudaError_t e;
            if ((e = plane_y(a, 0, grids.strip_y, st)) != cudaSuccess) return e;
            if ((e = plane_x(b, grids.strip_x, st)) != cudaSuccess) return e;
            return a.lens ? plane_y(b, 1, grids.strip_y, st) : cudaSuccess;
        } else {
            return launch_sweep(plane_kernel<NX, NY, CL, PB, SLO, PT>, nclusters * CL, PT, LC::SMEM, st, CL, a.overlap, a);
        }
    }

    static int max_clusters(const LaunchGrids& grids) {
        if constexpr (PL >= 2) {
            return grids.strip_y;   // CTAs of the y pass (clusters of one)
        } else {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(CL);
            cfg.blockDim = dim3(PT);
            cfg.dynamicSmemBytes = LC::SMEM;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = CL;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, plane_kernel<NX, NY, CL, PB, SLO, PT>, &cfg) != cudaSuccess) return 0;
            return n;
        }
    }

    static int pencil_blocks_per_sm() {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, pencil_kernel<NT, P, SLO, PM_EXIT_C128, CH>, TH, PC::SMEM) !=
            cudaSuccess)
            return 0;
        return n;
    }

    static constexpr int plane_smem() {
        if constexpr (PL == 5) return PlaneS::SMEM;
        else if constexpr (PL >= 2) return StripYCfg<NX, NY, CXS>::SMEM;
        else return LC::SMEM;
    }

    static const ShapeOps* ops() {
        static const ShapeOps o = {NX, NY, NT, P, SLO, CL, PB, PT, CH, LD, PL, LRB, NX * NY / SC::P, PC::SMEM, plane_smem(), &setup, &pencil, &plane,
                                   &max_clusters, &pencil_blocks_per_sm};
        return &o;
    }
};

}  // namespace mpc
