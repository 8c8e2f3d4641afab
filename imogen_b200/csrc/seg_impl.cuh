// Definitions of the launch entry points of the segment fluid and window magnet kernels declared in
// sweeps.cuh.  Each translation unit that includes this file instantiates them for one precision.
#pragma once

#include "launch.cuh"
#include "seg_fluid.cuh"
#include "seg_magnet.cuh"

namespace img {

// Segment fluid kernels by cells per thread: 2, 3, 4 and 8 (FP64: 2, 3 and 4); 3 serves pencils of 3 cells held
// whole by one thread.  Over a cluster (CLU) 2, 4 and 8 (FP64: 2 and 4), with fade ends 2 and 4.  FP64 CTAs
// of at most 256 threads have kernels of their own for 3 and 4 (MAXT, fluid_seg_kernel).
template <typename T, int MHD, bool CLU, bool FADE, int MAXT>
void (*fluid_seg_kernel_c(int C))(const FluidArgs) {
    if constexpr (sizeof(T) == 4 && !FADE) {
        if (C == 8) return fluid_seg_kernel<T, MHD, 8, VISC_NONE, CLU, FADE, MAXT>;
    }
    if constexpr (!CLU && !FADE) {
        if (C == 3) return fluid_seg_kernel<T, MHD, 3, VISC_NONE, CLU, FADE, MAXT>;
    }
    if constexpr (MAXT > 256) {
        if (C == 2) return fluid_seg_kernel<T, MHD, 2, VISC_NONE, CLU, FADE, MAXT>;
    }
    return fluid_seg_kernel<T, MHD, 4, VISC_NONE, CLU, FADE, MAXT>;
}

template <typename T, int MHD, bool CLU, bool FADE, int MAXT>
void (*fluid_seg_batch_kernel_c(int C))(const FluidArgs*, const BlockMap*) {
    if constexpr (sizeof(T) == 4 && !FADE) {
        if (C == 8) return fluid_seg_batch_kernel<T, MHD, 8, CLU, FADE, MAXT>;
    }
    if constexpr (!CLU && !FADE) {
        if (C == 3) return fluid_seg_batch_kernel<T, MHD, 3, CLU, FADE, MAXT>;
    }
    if constexpr (MAXT > 256) {
        if (C == 2) return fluid_seg_batch_kernel<T, MHD, 2, CLU, FADE, MAXT>;
    }
    return fluid_seg_batch_kernel<T, MHD, 4, CLU, FADE, MAXT>;
}

// With artificial viscosity: 2 and 4 cells per thread.
template <typename T, int MHD, int VT, int MAXT>
void (*fluid_seg_visc_kernel_c(int C))(const FluidArgs) {
    if constexpr (MAXT > 256) {
        if (C == 2) return fluid_seg_kernel<T, MHD, 2, VT, false, false, MAXT>;
    }
    return fluid_seg_kernel<T, MHD, 4, VT, false, false, MAXT>;
}

// Forms of the MHD fluxes (seg_flux): fade ends take form 2, artificial viscosity form 1, FP64 otherwise form 1 and
// the mixed form either.
template <typename T, int MHD, int MAXT>
void (*fluid_seg_kernel_m(int C, bool clu, bool fade, int visc))(const FluidArgs) {
    if constexpr (MHD < 2) {
        if (visc == VISC_NR) return fluid_seg_visc_kernel_c<T, MHD, VISC_NR, MAXT>(C);
        if (visc == VISC_CSW) return fluid_seg_visc_kernel_c<T, MHD, VISC_CSW, MAXT>(C);
    }
    if (fade) return fluid_seg_kernel_c<T, MHD ? 2 : 0, false, true, MAXT>(C);
    return clu ? fluid_seg_kernel_c<T, MHD, true, false, MAXT>(C) : fluid_seg_kernel_c<T, MHD, false, false, MAXT>(C);
}
template <typename T, int MAXT>
void (*fluid_seg_kernel_t(int C, int mhd, bool clu, bool fade, int visc))(const FluidArgs) {
    if constexpr (sizeof(T) == 4) {
        if (mhd == 2 && visc == VISC_NONE) return fluid_seg_kernel_m<T, 2, MAXT>(C, clu, fade, visc);
    }
    return mhd ? fluid_seg_kernel_m<T, 1, MAXT>(C, clu, fade, visc) : fluid_seg_kernel_m<T, 0, MAXT>(C, clu, fade, visc);
}
template <typename T>
void (*fluid_seg_kernel_p(int C, int mhd, bool clu, bool fade, int visc, unsigned block))(const FluidArgs) {
    if constexpr (sizeof(T) == 8) {
        if (block <= 256 && C > 2) return fluid_seg_kernel_t<T, 256>(C, mhd, clu, fade, visc);
    }
    return fluid_seg_kernel_t<T, 512>(C, mhd, clu, fade, visc);
}

template <typename T, int MHD, int MAXT>
void (*fluid_seg_batch_kernel_m(int C, bool clu, bool fade))(const FluidArgs*, const BlockMap*) {
    if (fade) return fluid_seg_batch_kernel_c<T, MHD ? 2 : 0, false, true, MAXT>(C);
    return clu ? fluid_seg_batch_kernel_c<T, MHD, true, false, MAXT>(C) : fluid_seg_batch_kernel_c<T, MHD, false, false, MAXT>(C);
}
template <typename T, int MAXT>
void (*fluid_seg_batch_kernel_t(int C, int mhd, bool clu, bool fade))(const FluidArgs*, const BlockMap*) {
    if constexpr (sizeof(T) == 4) {
        if (mhd == 2) return fluid_seg_batch_kernel_m<T, 2, MAXT>(C, clu, fade);
    }
    return mhd ? fluid_seg_batch_kernel_m<T, 1, MAXT>(C, clu, fade) : fluid_seg_batch_kernel_m<T, 0, MAXT>(C, clu, fade);
}
template <typename T>
void (*fluid_seg_batch_kernel_p(int C, int mhd, bool clu, bool fade, unsigned block))(const FluidArgs*, const BlockMap*) {
    if constexpr (sizeof(T) == 8) {
        if (block <= 256 && C > 2) return fluid_seg_batch_kernel_t<T, 256>(C, mhd, clu, fade);
    }
    return fluid_seg_batch_kernel_t<T, 512>(C, mhd, clu, fade);
}

template <typename T>
cudaError_t launch_fluid_seg(const FluidArgs& a, const PencilLaunch& L, int mhd) {
    return launch_pencil(fluid_seg_kernel_p<T>(L.seg, mhd, L.clu, L.fade, a.visc, L.block), a, L);
}
template <typename T>
cudaError_t launch_fluid_seg_batch(const FluidArgs* args, const BlockMap* map, const PencilLaunch& L, int mhd) {
    return launch_pencil_batch(fluid_seg_batch_kernel_p<T>(L.seg, mhd, L.clu, L.fade, L.block), args, map, L);
}

template <typename T>
cudaError_t fluid_seg_attributes(int optin) {
    for (int C : {2, 3, 4, 8}) {
        if (sizeof(T) == 8 && C == 8) continue;
        for (int mhd = 0; mhd < 3; ++mhd)
            for (int form = 0; form < 3; ++form) {   // plain, over a cluster, with fade ends
                if ((form == 1 && C == 3) || (form == 2 && C != 2 && C != 4)) continue;
                for (unsigned block : {256u, 512u}) {
                    if (block == 256 && (sizeof(T) == 4 || C == 2)) continue;   // the same kernels as 512's
                    cudaError_t e = allow_max_smem(fluid_seg_kernel_p<T>(C, mhd, form == 1, form == 2, VISC_NONE, block), optin);
                    if (e == cudaSuccess)
                        e = allow_max_smem(fluid_seg_batch_kernel_p<T>(C, mhd, form == 1, form == 2, block), optin);
                    for (int vt : {VISC_NR, VISC_CSW})
                        if (e == cudaSuccess && form == 0 && (C == 2 || C == 4))
                            e = allow_max_smem(fluid_seg_kernel_p<T>(C, mhd, false, false, vt, block), optin);
                    if (e != cudaSuccess) return e;
                }
            }
    }
    return cudaSuccess;
}

// Window magnet kernels by cells per thread (2, 3, 4, 8).
template <typename T>
void (*chain_win_kernel(int C))(const MagArgs) {
    if (C == 3) return mag_chain_win_kernel<T, 3>;
    return C == 2 ? mag_chain_win_kernel<T, 2> : (C == 8 ? mag_chain_win_kernel<T, 8> : mag_chain_win_kernel<T, 4>);
}
template <typename T>
void (*ct_win_kernel(int C))(const MagArgs) {
    if (C == 3) return mag_ct_win_kernel<T, 3>;
    return C == 2 ? mag_ct_win_kernel<T, 2> : (C == 8 ? mag_ct_win_kernel<T, 8> : mag_ct_win_kernel<T, 4>);
}
template <typename T>
void (*chain_win_batch_kernel(int C))(const MagArgs*, const BlockMap*) {
    if (C == 3) return mag_chain_win_batch_kernel<T, 3>;
    return C == 2 ? mag_chain_win_batch_kernel<T, 2> : (C == 8 ? mag_chain_win_batch_kernel<T, 8> : mag_chain_win_batch_kernel<T, 4>);
}
template <typename T>
void (*ct_win_batch_kernel(int C))(const MagArgs*, const BlockMap*) {
    if (C == 3) return mag_ct_win_batch_kernel<T, 3>;
    return C == 2 ? mag_ct_win_batch_kernel<T, 2> : (C == 8 ? mag_ct_win_batch_kernel<T, 8> : mag_ct_win_batch_kernel<T, 4>);
}

template <typename T>
cudaError_t launch_mag_chain_win(const MagArgs& a, const PencilLaunch& L) {
    return launch_pencil(chain_win_kernel<T>(L.seg), a, L);
}
template <typename T>
cudaError_t launch_mag_ct_win(const MagArgs& a, const PencilLaunch& L) {
    return launch_pencil(ct_win_kernel<T>(L.seg), a, L);
}
template <typename T>
cudaError_t launch_mag_chain_win_batch(const MagArgs* args, const BlockMap* map, const PencilLaunch& L) {
    return launch_pencil_batch(chain_win_batch_kernel<T>(L.seg), args, map, L);
}
template <typename T>
cudaError_t launch_mag_ct_win_batch(const MagArgs* args, const BlockMap* map, const PencilLaunch& L) {
    return launch_pencil_batch(ct_win_batch_kernel<T>(L.seg), args, map, L);
}

// The window chain kernels' exchange planes (chain_win_smem_bytes) can exceed the default limit.
template <typename T>
cudaError_t chain_win_attributes(int optin) {
    for (int C : {2, 3, 4, 8}) {
        cudaError_t e = allow_max_smem(chain_win_kernel<T>(C), optin);
        if (e == cudaSuccess) e = allow_max_smem(chain_win_batch_kernel<T>(C), optin);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace img
