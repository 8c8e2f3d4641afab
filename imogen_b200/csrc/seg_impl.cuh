// Definitions of the launch entry points of the segment fluid and window magnet kernels declared in
// sweeps.cuh.  Each translation unit that includes this file instantiates them for one precision.
#pragma once

#include "launch.cuh"
#include "seg_fluid.cuh"
#include "seg_magnet.cuh"

namespace img {

// Segment fluid kernels by cells per thread (2, 3, 4 and 8; FP64: 2, 3 and 4).  3 serves pencils of
// 3 cells held whole by one thread.
template <typename T, bool MHD>
void (*fluid_seg_kernel_c(int C))(const FluidArgs) {
    if constexpr (sizeof(T) == 4) {
        if (C == 8) return fluid_seg_kernel<T, MHD, 8>;
    }
    if (C == 3) return fluid_seg_kernel<T, MHD, 3>;
    return C == 2 ? fluid_seg_kernel<T, MHD, 2> : fluid_seg_kernel<T, MHD, 4>;
}

template <typename T, bool MHD>
void (*fluid_seg_batch_kernel_c(int C))(const FluidArgs*, const BlockMap*) {
    if constexpr (sizeof(T) == 4) {
        if (C == 8) return fluid_seg_batch_kernel<T, MHD, 8>;
    }
    if (C == 3) return fluid_seg_batch_kernel<T, MHD, 3>;
    return C == 2 ? fluid_seg_batch_kernel<T, MHD, 2> : fluid_seg_batch_kernel<T, MHD, 4>;
}

// With artificial viscosity: 2 and 4 cells per thread.
template <typename T, bool MHD, int VT>
void (*fluid_seg_visc_kernel_c(int C))(const FluidArgs) {
    return C == 2 ? fluid_seg_kernel<T, MHD, 2, VT> : fluid_seg_kernel<T, MHD, 4, VT>;
}

template <typename T>
void (*fluid_seg_kernel_p(int C, bool mhd, int visc = VISC_NONE))(const FluidArgs) {
    if (visc == VISC_NR) return mhd ? fluid_seg_visc_kernel_c<T, true, VISC_NR>(C) : fluid_seg_visc_kernel_c<T, false, VISC_NR>(C);
    if (visc == VISC_CSW) return mhd ? fluid_seg_visc_kernel_c<T, true, VISC_CSW>(C) : fluid_seg_visc_kernel_c<T, false, VISC_CSW>(C);
    return mhd ? fluid_seg_kernel_c<T, true>(C) : fluid_seg_kernel_c<T, false>(C);
}

template <typename T>
void (*fluid_seg_batch_kernel_p(int C, bool mhd))(const FluidArgs*, const BlockMap*) {
    return mhd ? fluid_seg_batch_kernel_c<T, true>(C) : fluid_seg_batch_kernel_c<T, false>(C);
}

// Cluster (CLU) forms of the segment fluid kernel: 2, 4 and 8 cells per thread (FP64: 2 and 4).
template <typename T, bool MHD>
void (*fluid_seg_clu_kernel_c(int C))(const FluidArgs) {
    if constexpr (sizeof(T) == 4) {
        if (C == 8) return fluid_seg_clu_kernel<T, MHD, 8>;
    }
    return C == 2 ? fluid_seg_clu_kernel<T, MHD, 2> : fluid_seg_clu_kernel<T, MHD, 4>;
}

template <typename T, bool MHD>
void (*fluid_seg_clu_batch_kernel_c(int C))(const FluidArgs*, const BlockMap*) {
    if constexpr (sizeof(T) == 4) {
        if (C == 8) return fluid_seg_clu_batch_kernel<T, MHD, 8>;
    }
    return C == 2 ? fluid_seg_clu_batch_kernel<T, MHD, 2> : fluid_seg_clu_batch_kernel<T, MHD, 4>;
}

template <typename T>
void (*fluid_seg_clu_kernel_p(int C, bool mhd))(const FluidArgs) {
    return mhd ? fluid_seg_clu_kernel_c<T, true>(C) : fluid_seg_clu_kernel_c<T, false>(C);
}

template <typename T>
void (*fluid_seg_clu_batch_kernel_p(int C, bool mhd))(const FluidArgs*, const BlockMap*) {
    return mhd ? fluid_seg_clu_batch_kernel_c<T, true>(C) : fluid_seg_clu_batch_kernel_c<T, false>(C);
}

template <typename T>
cudaError_t launch_fluid_seg(const FluidArgs& a, const PencilLaunch& L, bool mhd) {
    if (L.clu) return launch_pencil(fluid_seg_clu_kernel_p<T>(L.seg, mhd), a, L);
    return launch_pencil(fluid_seg_kernel_p<T>(L.seg, mhd, a.visc), a, L);
}
template <typename T>
cudaError_t launch_fluid_seg_batch(const FluidArgs* args, const BlockMap* map, const PencilLaunch& L, bool mhd) {
    if (L.clu) return launch_pencil_batch(fluid_seg_clu_batch_kernel_p<T>(L.seg, mhd), args, map, L);
    return launch_pencil_batch(fluid_seg_batch_kernel_p<T>(L.seg, mhd), args, map, L);
}

template <typename T>
cudaError_t fluid_seg_attributes(int optin) {
    for (int C : {2, 3, 4, 8}) {
        if (sizeof(T) == 8 && C == 8) continue;
        for (int mhd = 0; mhd < 2; ++mhd) {
            cudaError_t e = allow_max_smem(fluid_seg_kernel_p<T>(C, mhd != 0), optin);
            if (e == cudaSuccess) e = allow_max_smem(fluid_seg_batch_kernel_p<T>(C, mhd != 0), optin);
            for (int vt : {VISC_NR, VISC_CSW})
                if (e == cudaSuccess && (C == 2 || C == 4)) e = allow_max_smem(fluid_seg_kernel_p<T>(C, mhd != 0, vt), optin);
            if (e == cudaSuccess && C != 3) e = allow_max_smem(fluid_seg_clu_kernel_p<T>(C, mhd != 0), optin);
            if (e == cudaSuccess && C != 3) e = allow_max_smem(fluid_seg_clu_batch_kernel_p<T>(C, mhd != 0), optin);
            if (e != cudaSuccess) return e;
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
