// Segment form of the fused fluid sweep (fluid/relaxingFluid.m:16-73, fluid/wFluidFlux.m:14-44,
// pressure/pressure.m:23-64, flux/*Limiter.m) for pencils with circ, const or fade ends.
//
// Each thread owns C consecutive cells of a pencil (a "segment"; the last one may be shorter), so every
// stencil neighbour inside a segment is a register; only the cells at the two ends of a segment are
// exchanged, through shared memory, and the exchanges ride on the two barriers that the pencil maxima
// need anyway:
//   stage 1  load the segment (128-bit loads along x), 'totsnd' pressure, freezing-speed candidate and
//            the flux numerators F (w = F / c_f) of every cell; publish (u, F) of the first and last
//            cell; barrier; c_f = pencil max.
//   stage 2  predictor half step (relaxingFluid.m:30-39); pressure, speed and F of the half-step state;
//            publish (u*, F*) of the first two and last two cells; barrier; c_f* = pencil max.
//   stage 3  corrector fluxes over the segment and the two neighbour cells each side, the TVD limiter
//            (relaxingFluid.m:57-62) -- the limited values of the neighbour cells next to the segment are
//            computed here as well, from the published cells -- and the update (relaxingFluid.m:64-71);
//            store; fused CFL maxima on the last sweep of a step.
// R = (u + F/c_f)/2 and L = (u - F/c_f)/2 take one FMA each (the predictor leaves the 2 to the update).  In the mixed
// form two variables at a time go through the packed FP32 instructions (lanes.cuh).
// Fade ends (fade_shift.m) blend every shifted array near the ends toward the shifted end values: those
// launches (FADE) form the shifted values cell by cell, take the ends' rows from a small anchor set and
// exchange the limited fluxes behind one more barrier.
// With artificial viscosity (fluid/ArtificialViscosity.m) stages 1 and 2 each publish the viscosity
// exchange set with the pencil maximum, then compute the viscous pressure and F and publish (u, F)
// behind one more barrier: four barriers instead of two.
// Per cell the operations are those of the pencil-tile kernels (fluid_sweep.cuh) in the same order; the momentum
// and cell-centred B are held in sweep-rotated order (the component along the sweep first).  The FMAs are written
// out (the unit is compiled without implicit ones), so within one form of the fluxes results do not depend on the
// tiling.  MHD = 2 sums and rounds the B terms of the fluxes as the pencil-tile kernels do, MHD = 1 in rotated order
// (seg_flux); the launch picks the form.
//
// Thread placement (SweepGeom with G = S segments per pencil, RC = N): along x the S threads of a
// pencil are consecutive (thread t = b*S + s), along y and z the Wb pencils of the CTA are (t = s*Wb +
// b), so global loads and stores stay coalesced along x; threads past the last segment idle.  A pencil
// along x may span the CTAs of a cluster (CLU; segment s = rank*NT + t), whose exchanges then read the
// neighbours' shared memory through DSMEM.  Pencil ends: a circ end's neighbour is the pencil's other end;
// a const (or fade) end's ghost is the end cell itself (constant_shift.m), applied to every shifted array,
// the limited fluxes included.
#pragma once

#include <type_traits>

#include "fluid_sweep.cuh"
#include "lanes.cuh"

namespace img {

// FP64 words per thread of the artificial-viscosity exchange set (seg_visc_publish).
constexpr int VISC_ROWS = 9;

// Shared memory: per thread the exchange records, (u, F) of 2 cells and (u*, F*) of 4 cells, 10 values
// each; two pencil maxima per pencil; then the FP64 viscosity exchange set, or with fade ends the anchors
// (4 rows of 10 values per pencil and stage, 4 of 5 for the limited fluxes).
template <typename T>
__host__ __device__ inline size_t seg_fluid_smem_bytes(int NT, int Wb, bool visc = false, bool fade = false) {
    return sizeof(T) * (size_t)60 * NT + 16 * (size_t)Wb + (visc ? sizeof(double) * VISC_ROWS * NT : 0) +
           (fade ? sizeof(T) * (size_t)100 * Wb : 0);
}

// Placement of one thread in the segment layout.
struct SegPos {
    int b, s;            // pencil within the CTA, segment within the pencil
    int rank;            // cluster rank (one pencil per cluster)
    bool colok;          // the pencil exists (the last CTA may hold fewer than Wb) and so does the segment
    int base;            // offset of the pencil's row 0 (grids have fewer than 2^31 cells)
    template <bool CLU>
    __device__ __forceinline__ void init(const SweepGeom& g, unsigned vblock) {
        int t = threadIdx.x;
        unsigned blk = vblock;
        rank = 0;
        if constexpr (CLU) {   // one pencil over the CL CTAs of a cluster (CL = 1: one CTA)
            blk = g.div_cl.div(vblock);
            rank = (int)(vblock - blk * (unsigned)g.CL);
            b = 0;
            s = t + rank * g.NT;
        } else {
            const unsigned q = g.div_lanes.div((unsigned)t);   // t / S (x) or t / Wb (y, z)
            if (g.d == 0) { b = (int)q; s = t - b * g.G; }
            else { s = (int)q; b = t - s * g.Wb; }
        }
        const int col = (int)(blk * (unsigned)g.Wb + (unsigned)b);
        colok = col < (int)g.ncol && b < g.Wb && s < g.G;
        const unsigned c = colok ? (unsigned)col : 0u;
        const int c2 = (int)g.div_n1.div(c);
        const int c1 = (int)(c - (unsigned)c2 * (unsigned)g.n1);
        base = c1 * (int)g.s1 + c2 * (int)g.s2;
    }
};

// C consecutive values of array p starting at offset o, stride sd (vector loads when sd == 1: the
// offset is a multiple of C and arrays start 256-byte aligned).
template <typename T, int C>
__device__ __forceinline__ void seg_load(const void* p, long long o, long long sd, bool vec, T (&out)[C]) {
    const T* a = reinterpret_cast<const T*>(p) + o;
    if (vec) {
        if constexpr (sizeof(T) == 4 && C % 4 == 0) {
#pragma unroll
            for (int k = 0; k < C; k += 4) {
                const float4 v = *reinterpret_cast<const float4*>(a + k);
                out[k] = v.x; out[k + 1] = v.y; out[k + 2] = v.z; out[k + 3] = v.w;
            }
            return;
        } else if constexpr (C % 2 == 0) {
            using V2 = typename std::conditional<sizeof(T) == 4, float2, double2>::type;
#pragma unroll
            for (int k = 0; k < C; k += 2) {
                const V2 v = *reinterpret_cast<const V2*>(a + k);
                out[k] = v.x; out[k + 1] = v.y;
            }
            return;
        }
    }
#pragma unroll
    for (int k = 0; k < C; ++k) out[k] = a[(long long)k * sd];
}

template <typename T, int C>
__device__ __forceinline__ void seg_store(void* p, long long o, long long sd, bool vec, const T (&v)[C]) {
    T* a = reinterpret_cast<T*>(p) + o;
    if (vec) {
        if constexpr (sizeof(T) == 4 && C % 4 == 0) {
#pragma unroll
            for (int k = 0; k < C; k += 4) *reinterpret_cast<float4*>(a + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
            return;
        } else if constexpr (C % 2 == 0) {
#pragma unroll
            for (int k = 0; k < C; k += 2) {
                if constexpr (sizeof(T) == 4) *reinterpret_cast<float2*>(a + k) = make_float2(v[k], v[k + 1]);
                else *reinterpret_cast<double2*>(a + k) = make_double2(v[k], v[k + 1]);
            }
            return;
        }
    }
#pragma unroll
    for (int k = 0; k < C; ++k) a[(long long)k * sd] = v[k];
}

// Own cells of an array: vector accesses where the segments allow (vec), else cell by cell; past the
// pencil's end (a ragged last segment, idle threads) `fill`, and nothing stored.
// ONCE: the strided cells of y and z sweeps are loaded past the L1 cache (nobody reads them again, and their
// 32-byte rows would each take a 128-byte line from what does come back).
template <typename T, int C, bool ONCE = false>
__device__ __forceinline__ void win_load(const void* ptr, int o, int sd, bool vec, int nown, T fill, T (&out)[C]) {
    const T* p = reinterpret_cast<const T*>(ptr);
    if (vec && nown == C) {
        seg_load<T, C>(p, o, 1, true, out);
    } else if (ONCE && sd != 1) {
#pragma unroll
        for (int k = 0; k < C; ++k) out[k] = k < nown ? __ldcg(p + (o + k * sd)) : fill;
    } else {
#pragma unroll
        for (int k = 0; k < C; ++k) out[k] = k < nown ? p[o + k * sd] : fill;
    }
}
template <typename T, int C>
__device__ __forceinline__ void win_store(void* ptr, int o, int sd, bool vec, int nown, const T (&v)[C]) {
    T* p = reinterpret_cast<T*>(ptr);
    if (vec && nown == C) {
        seg_store<T, C>(p, o, 1, true, v);
    } else {
#pragma unroll
        for (int k = 0; k < C; ++k)
            if (k < nown) p[o + k * sd] = v[k];
    }
}

// Constants of the 'totsnd' pressure (pressure.m:23-64) from gamma.
struct SegPressure {
    double half_g, g1, half_g1, p_ms;
    __device__ __forceinline__ explicit SegPressure(double G)
        : half_g(0.5 * G), g1(G - 1.0), half_g1((G - 1.0) * 0.5), p_ms(0.5 * (2.0 - G)) {}
    // P and rho c_s^2 / 2 from x = E - rho v^2/2 and msq = B^2.  Each B^2 term is rounded before it joins (G-1) x, as
    // the pencil-tile kernels' pressure_totsnd_mixed comes out, whose FP64 bits the mixed form shares: one of the
    // other orders differs in the last FP64 bit of every other cell, hence in the FP32 pressure of one in 2e9, and a
    // 256^3 shear run grows that to 1e-3 of B's scale at single cells in 120 iterations.
    template <int MSQ>
    __device__ __forceinline__ void totals(double x, double msq, double& pt, double& hc2) const {
        if constexpr (MSQ) {
            hc2 = fma(half_g, fma(g1, x, -(half_g1 * msq)), msq);
            pt = fma(g1, x, p_ms * msq);
        } else {
            pt = g1 * x;
            hc2 = half_g * pt;
        }
    }
};

// 'totsnd' pressure, sound speed, 1/rho and the freezing-speed candidate |p_X / rho| + c_s of one cell
// (rotated order; msq = B^2 of the cell-centred components without isZero).  Mixed form: FP64 throughout,
// with 1/rho from the one-instruction FP32 estimate refined by one FP64 Newton step; the sound speed's
// square root is taken in FP32.
template <int MSQ>
__device__ __forceinline__ float seg_pressure(const SegPressure& k, const float (&u)[5], double msq, float& p, float& cs,
                                              float& ir) {
    ir = rcp_approx(u[0]);
    const double e0 = (double)ir;
    const double inv = e0 * fma(-(double)u[0], e0, 2.0);
    const double px = u[1], py = u[2], pz = u[3];
    const double psq = fma(pz, pz, fma(px, px, py * py));
    double hc2, pt;
    k.totals<MSQ>(fma(-(0.5 * psq), inv, (double)u[4]), msq, pt, hc2);
    cs = sqrt_approx(fabsf(2.f * (float)(hc2 * inv)));
    p = pt < 0 ? 0.f : (float)pt;
    return fabsf(u[1] * ir) + cs;
}
template <int MSQ>
__device__ __forceinline__ double seg_pressure(const SegPressure& k, const double (&u)[5], double msq, double& p, double& cs,
                                               double& ir) {
    ir = recip(u[0]);
    const double psq = fma(u[3], u[3], fma(u[1], u[1], u[2] * u[2]));
    double hc2, pt;
    k.totals<MSQ>(fma(-(0.5 * psq), ir, u[4]), msq, pt, hc2);
    cs = sqrt_goldschmidt(fabs(2.0 * (hc2 * ir)));
    p = pt < 0 ? 0.0 : pt;
    return fabs(u[1] * ir) + cs;
}

// The flux numerators F of wFluidFlux.m:31-44 (w = F / c_f) for one cell (rotated order).  MHD = 2: B.p is summed in
// the order x, y, z, and the transverse momentum fluxes round v p before they take B B off it, as the pencil-tile
// kernels do; MHD = 1: B.p in rotated order, B B rounded first.
template <typename T, int MHD>
__device__ __forceinline__ void seg_flux(int d, bool tile, const T (&u)[5], const T (&bb)[3], T press, T ir, T (&F)[5]) {
    const T velocity = u[1] * ir;
    F[0] = u[1];
    if constexpr (MHD) {
        T dot;
        if (MHD == 1 || d == 0) dot = v_fma(bb[2], u[3], v_fma(bb[0], u[1], bb[1] * u[2]));
        else if (d == 1) dot = v_fma(bb[2], u[3], v_fma(bb[1], u[2], bb[0] * u[1]));
        else dot = v_fma(bb[0], u[1], v_fma(bb[1], u[2], bb[2] * u[3]));
        F[4] = v_fma(velocity, u[4] + press, -((bb[0] * dot) * ir));
        if (MHD == 2) F[1] = v_fma(-bb[0], bb[0], velocity * u[1] + press);
        else F[1] = v_fma(velocity, u[1], press) - bb[0] * bb[0];
        F[2] = MHD == 2 ? v_fma(-bb[0], bb[1], velocity * u[2]) : v_fma(velocity, u[2], -(bb[0] * bb[1]));
        F[3] = MHD == 2 ? v_fma(-bb[0], bb[2], velocity * u[3]) : v_fma(velocity, u[3], -(bb[0] * bb[2]));
    } else {
        F[4] = velocity * (u[4] + press);
        F[1] = tile ? velocity * u[1] + press : v_fma(velocity, u[1], press);
        F[2] = velocity * u[2];
        F[3] = velocity * u[3];
    }
}

// ---- artificial viscosity (fluid/ArtificialViscosity.m) in the segment layout ---------------------
// Computed in FP64 for both forms, with explicit round-to-nearest products and sums (no FMA
// contraction), in the reference's operation order.  The stage's state is the one wFluidFlux.m
// receives: the primaries for the predictor, the half-step stores for the corrector; the viscous term
// is added to the 'totsnd' pressure after the freezing speed is taken (wFluidFlux.m:18-24).

// cswSoundSpeed's per-cell sound speed (ArtificialViscosity.m:157-190) from the natural-order
// momentum and cell-centred B of one cell.  As the reference writes it, only the z momentum of the
// velocity-squared sum is divided by rho^2, and every B component counts (no isZero test).
__device__ __forceinline__ double csw_cell_sound(double G, double rho, double px, double py, double pz, double E,
                                                 double bx, double by, double bz) {
    const double vel_sq = __dadd_rn(__dadd_rn(__dmul_rn(px, px), __dmul_rn(py, py)), __dmul_rn(pz, pz) / __dmul_rn(rho, rho));
    const double mag_sq = __dadd_rn(__dadd_rn(__dmul_rn(bx, bx), __dmul_rn(by, by)), __dmul_rn(bz, bz));
    double s = __dmul_rn(G - 1.0, __dsub_rn(E, __dmul_rn(__dmul_rn(0.5, rho), vel_sq)));
    s = __dsub_rn(s, __dmul_rn(__dmul_rn(G - 1.0, 0.5), mag_sq));
    return sqrt(fabs(__dadd_rn(__dmul_rn(G, s), __dmul_rn(2.0, mag_sq)) / rho));
}

// Per-cell viscosity inputs of one stage and their exchange set V ([VISC_ROWS][NT] FP64): v = p_X/rho
// of cells 0, 1, C-2, C-1 (rows 0-3), rho of cells 0 and C-1 (rows 4-5), the CSW cell sound speed of
// cells 0 and C-1 (rows 6-7) and p_X of cell 0 (row 8).  w holds the stage state in sweep-rotated order;
// (nx, ny, nz) give the rotated slot (0-2) of the natural components.
template <typename T, int C, int VT>
__device__ __forceinline__ void seg_visc_publish(const T (&w)[5][C], const T (&bb)[3][C], double G, int nx, int ny, int nz,
                                                 double* V, int NT, int t, double (&vel)[C], double (&snd)[C]) {
    static_assert(C >= 2, "the viscosity stencil reaches 2 cells: at least 2 cells per thread");
#pragma unroll
    for (int k = 0; k < C; ++k) {
        vel[k] = (double)w[1][k] / (double)w[0][k];
        if constexpr (VT == VISC_CSW) {
            const double p[3] = {(double)w[1][k], (double)w[2][k], (double)w[3][k]};
            const double b[3] = {(double)bb[0][k], (double)bb[1][k], (double)bb[2][k]};
            auto pick = [](const double (&a)[3], int s) { return s == 0 ? a[0] : (s == 1 ? a[1] : a[2]); };
            snd[k] = csw_cell_sound(G, (double)w[0][k], pick(p, nx), pick(p, ny), pick(p, nz), (double)w[4][k],
                                    pick(b, nx), pick(b, ny), pick(b, nz));
        } else {
            snd[k] = 0.0;
        }
    }
    if constexpr (VT == VISC_CSW) {
        V[0 * NT + t] = vel[0];
        V[1 * NT + t] = vel[1];
        V[2 * NT + t] = vel[C - 2];
        V[3 * NT + t] = vel[C - 1];
        V[4 * NT + t] = (double)w[0][0];
        V[5 * NT + t] = (double)w[0][C - 1];
        V[6 * NT + t] = snd[0];
        V[7 * NT + t] = snd[C - 1];
    } else {
        V[8 * NT + t] = (double)w[1][0];
    }
}

// The viscous pressure q of the C own cells (after the barrier that follows seg_visc_publish).  lt/rt:
// the threads of the neighbour segments; lo_own/hi_own: a const pencil end (its ghosts are the end
// cell, constant_shift.m); cs: the 'totsnd' sound speed of each cell (Neumann-Richtmyer).
template <typename T, int C, int VT>
__device__ __forceinline__ void seg_visc_terms(const FluidArgs& a, double G, const T (&w)[5][C], const T (&cs)[C],
                                               const double (&vel)[C], const double (&snd)[C], const double* V, int NT,
                                               int lt, int rt, bool lo_own, bool hi_own, double (&q)[C]) {
    if constexpr (VT == VISC_NR) {
        // viscousMagnitude = min(p_X.shift(X, 1) - p_X, 0); q = vm (c1 c_s + c2 vm / rho)
#pragma unroll
        for (int k = 0; k < C; ++k) {
            const double pn = k + 1 < C ? (double)w[1][k + 1] : (hi_own ? (double)w[1][C - 1] : V[8 * NT + rt]);
            const double vm = fmin(__dsub_rn(pn, (double)w[1][k]), 0.0);
            q[k] = __dmul_rn(vm, __dadd_rn(__dmul_rn(a.vc1, (double)cs[k]), __dmul_rn(a.vc2, vm) / (double)w[0][k]));
        }
    } else {
        double vv[C + 4], rr[C + 2], ss[C + 2];   // cells -2 .. C+1 and -1 .. C
#pragma unroll
        for (int k = 0; k < C; ++k) {
            vv[k + 2] = vel[k];
            rr[k + 1] = (double)w[0][k];
            ss[k + 1] = snd[k];
        }
        vv[1] = lo_own ? vel[0] : V[3 * NT + lt];
        vv[0] = lo_own ? vel[0] : V[2 * NT + lt];
        rr[0] = lo_own ? rr[1] : V[5 * NT + lt];
        ss[0] = lo_own ? ss[1] : V[7 * NT + lt];
        vv[C + 2] = hi_own ? vel[C - 1] : V[0 * NT + rt];
        vv[C + 3] = hi_own ? vel[C - 1] : V[1 * NT + rt];
        rr[C + 1] = hi_own ? rr[C] : V[4 * NT + rt];
        ss[C + 1] = hi_own ? ss[C] : V[6 * NT + rt];
#pragma unroll
        for (int k = 0; k < C; ++k) {
            const double mb = rr[k], mc = rr[k + 2];
            const double rho = __dmul_rn(__dmul_rn(2.0, mc), mb) / __dadd_rn(mc, mb);   // averaged density
            const double c = fmax(fmin(ss[k], ss[k + 2]), 0.0);                           // cswSoundSpeed
            const double v0 = vv[k], v1 = vv[k + 1], v2 = vv[k + 3], v3 = vv[k + 4];
            const double dv = __dsub_rn(v2, v1);
            const double rl = __dsub_rn(v3, v2) / __dmul_rn(2.0, dv);
            const double rr_ = __dsub_rn(v1, v0) / __dmul_rn(2.0, dv);
            const double lim = fmax(0.0, fmin(fmin(__dmul_rn(0.5, __dadd_rn(rl, rr_)),
                                                   fmin(__dmul_rn(2.0, rl), __dmul_rn(2.0, rr_))), 1.0));
            const double adv = fabs(dv);
            const double root = sqrt(__dadd_rn(__dmul_rn(a.vk2, __dmul_rn(dv, dv)), __dmul_rn(a.vc1sq, __dmul_rn(c, c))));
            const double mag = __dadd_rn(__dmul_rn(a.vk1, adv) / 4.0, root);
            q[k] = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(dv < 0.0 ? 1.0 : 0.0, rho), mag), __dsub_rn(1.0, lim)), adv);
        }
    }
}

// press + viscosity.solve: in FP64 the reference's sum; in the mixed form the FP32 pressure plus the
// rounded viscous term.
template <typename T>
__device__ __forceinline__ T visc_add(T p, double q) {
    if constexpr (sizeof(T) == 4) return p + (float)q;
    else return __dadd_rn(p, q);
}

// ---- exchange records ---------------------------------------------------------------------------------
// The 10 values (u, F) of one cell, `slots` records per thread, in parts by the variables that are worked on
// together: 16 bytes of (u, F) of two FP32 variables or one FP64 variable (8 for the fifth FP32 one), the same
// part of consecutive threads' records on consecutive 16 bytes.
template <typename T>
__host__ __device__ constexpr int seg_rec_bytes() { return 10 * (int)sizeof(T); }

__device__ __forceinline__ void rec_put(unsigned char* X, int slots, int slot, int NT, int t, const float (&u)[5],
                                        const float (&F)[5]) {
    const int i = slot * NT + t, n = slots * NT;
    reinterpret_cast<float4*>(X)[i] = make_float4(u[0], u[1], F[0], F[1]);
    reinterpret_cast<float4*>(X)[n + i] = make_float4(u[2], u[3], F[2], F[3]);
    reinterpret_cast<float2*>(X)[4 * n + i] = make_float2(u[4], F[4]);
}
__device__ __forceinline__ void rec_put(unsigned char* X, int slots, int slot, int NT, int t, const double (&u)[5],
                                        const double (&F)[5]) {
    const int i = slot * NT + t, n = slots * NT;
    double2* P = reinterpret_cast<double2*>(X);
#pragma unroll
    for (int v = 0; v < 5; ++v) P[v * n + i] = make_double2(u[v], F[v]);
}
// Variables v .. v + M - 1 (one part) of record i.
template <int v, int M>
__device__ __forceinline__ void rec_part(const unsigned char* X, int slots, int i, int NT, float (&u)[M], float (&F)[M]) {
    const int n = slots * NT;
    if constexpr (M == 2) {
        const float4 a = reinterpret_cast<const float4*>(X)[(v / 2) * n + i];
        u[0] = a.x; u[1] = a.y; F[0] = a.z; F[1] = a.w;
    } else {
        static_assert(v == 4, "the fifth variable stands alone");
        const float2 a = reinterpret_cast<const float2*>(X)[4 * n + i];
        u[0] = a.x; F[0] = a.y;
    }
}
template <int v, int M>
__device__ __forceinline__ void rec_part(const unsigned char* X, int slots, int i, int NT, double (&u)[M], double (&F)[M]) {
    static_assert(M == 1, "FP64 variables go one by one");
    const double2 a = reinterpret_cast<const double2*>(X)[v * slots * NT + i];
    u[0] = a.x; F[0] = a.y;
}
__device__ __forceinline__ void rec_get(const unsigned char* X, int slots, int i, int NT, float (&u)[5], float (&F)[5]) {
    float a[2], b[2], c[1], d[1];
    rec_part<0, 2>(X, slots, i, NT, a, b);
    u[0] = a[0]; u[1] = a[1]; F[0] = b[0]; F[1] = b[1];
    rec_part<2, 2>(X, slots, i, NT, a, b);
    u[2] = a[0]; u[3] = a[1]; F[2] = b[0]; F[3] = b[1];
    rec_part<4, 1>(X, slots, i, NT, c, d);
    u[4] = c[0]; F[4] = d[0];
}
__device__ __forceinline__ void rec_get(const unsigned char* X, int slots, int i, int NT, double (&u)[5], double (&F)[5]) {
    const int n = slots * NT;
    const double2* P = reinterpret_cast<const double2*>(X);
#pragma unroll
    for (int v = 0; v < 5; ++v) {
        const double2 a = P[v * n + i];
        u[v] = a.x;
        F[v] = a.y;
    }
}

// One neighbour's record: the exchange sets it lies in (another CTA's across a cluster) and its index.
struct SegRef {
    const unsigned char *X1, *X2;
    int i1, i2;
};

// ---- pencil maxima ------------------------------------------------------------------------------------
// Maximum of non-negative speeds over a pencil, kept as ordered bits per pencil in shared memory (zeroed
// before the first barrier): each warp reduces what it can, then one shared atomic per pencil and warp
// (per lane where a warp holds many short pencils).  One value to read after the barrier, where a table of
// warp maxima took up to 16 loads and compares in every thread.
__device__ __forceinline__ void seg_max_bits(unsigned* m, float v) { atomicMax(m, __float_as_uint(v + 0.0f)); }
__device__ __forceinline__ void seg_max_bits(unsigned long long* m, double v) {
    atomicMax(m, (unsigned long long)__double_as_longlong(v + 0.0));
}
template <typename T> struct SegBits { using U = unsigned long long; };
template <> struct SegBits<float> { using U = unsigned; };
__device__ __forceinline__ float seg_from_bits(unsigned b) { return __uint_as_float(b); }
__device__ __forceinline__ double seg_from_bits(unsigned long long b) { return __longlong_as_double((long long)b); }

template <typename T, bool CLU>
__device__ __forceinline__ void seg_max_publish(const SweepGeom& g, const SegPos& sp, T v, typename SegBits<T>::U* m) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    if (!CLU && g.G == 1) return;
    if (CLU || (g.d == 0 && (g.G & 31) == 0)) {         // a warp's lanes belong to one pencil
        v = warp_max_nonneg(v);
        if (lane == 0 && sp.b < g.Wb) seg_max_bits(m + sp.b, v);
    } else if (g.d != 0) {                               // lanes b, b + Wb, ... belong to pencil b
        for (int o = 16; o >= g.Wb; o >>= 1) v = fmax(v, __shfl_xor_sync(full, v, o));
        if (lane < g.Wb) seg_max_bits(m + sp.b, v);
    } else {                                             // along x, segment counts of any size
        const int b0 = __shfl_sync(full, sp.b, 0), b1 = __shfl_sync(full, sp.b, 31);
        if (b0 == b1) {
            v = warp_max_nonneg(v);
            if (lane == 0 && sp.b < g.Wb) seg_max_bits(m + sp.b, v);
        } else if (sp.b < g.Wb) {
            seg_max_bits(m + sp.b, v);
        }
    }
}
template <typename T, bool CLU>
__device__ __forceinline__ T seg_max_collect(const SweepGeom& g, const SegPos& sp, T own, typename SegBits<T>::U* m) {
    if (!CLU && g.G == 1) return own;
    if (CLU && g.CL > 1) {
        T c = T(0);
        for (int r = 0; r < g.CL; ++r) c = fmax(c, seg_from_bits(*cg::this_cluster().map_shared_rank(m, r)));
        return c;
    }
    return seg_from_bits(m[sp.b < g.Wb ? sp.b : 0]);
}

// Stage barrier of the segment kernel: the cluster's where a pencil spans a cluster.
template <bool CLU>
__device__ __forceinline__ void sp_sync(const SweepGeom& g) {
    if (CLU && g.CL > 1) cluster_sync();
    else __syncthreads();
}

// ---- predictor and corrector of one lane of variables --------------------------------------------------
// Which of a segment's cells round the change of the half step before they add it (FluidArgs.round_cells = n: a
// pencil's cells n - 1, 2 n - 1, ..., the energy excepted), among the last one and the fourth of 8 (any of 3): 0 none,
// 1 yes, 2 as the launch says (round_cells is 4 in form 1 of the MHD fluxes wherever C is a multiple of 4, and 0 in
// form 2).
template <typename T, int MHD, int C>
__host__ __device__ constexpr int seg_round_mode() {
    return sizeof(T) == 8 || MHD == 2 ? 0 : (MHD == 1 && C % 4 == 0 ? 1 : 2);
}

// Predictor (relaxingFluid.m:30-39): u and F at cells -1 .. C (index j + 1); ic = 1 / c_f, h = dt/dx c_f / 4.
template <typename V, int C, int RND>
__device__ __forceinline__ void seg_predict(const V (&u)[C + 2], const V (&F)[C + 2], V ic, V nic, V h, V nh, unsigned round,
                                            V (&us)[C]) {
    V R[C + 1], L[C + 1];   // 2R at cells -1 .. C-1 (j + 1), 2L at cells 0 .. C (j)
#pragma unroll
    for (int j = 0; j <= C; ++j) {
        R[j] = v_fma(F[j], ic, u[j]);
        L[j] = v_fma(F[j + 1], nic, u[j + 1]);
    }
#pragma unroll
    for (int k = 0; k < C; ++k) {
        const V S = v_sub(v_add(v_sub(R[k + 1], R[k]), L[k]), L[k + 1]);
        // (a product of pairs and a sum of pairs become one FMA; v_sub is an FMA itself, which keeps them apart)
        if (RND == 1 && (k == C - 1 || k % 4 == 3)) {
            us[k] = v_sub(u[k + 1], v_mul(h, S));
        } else {
            us[k] = v_fma(nh, S, u[k + 1]);
            if (RND == 2 && (C == 3 || k == C - 1 || k % 4 == 3))
                us[k] = v_pick(round >> k & 1, v_sub(u[k + 1], v_mul(h, S)), us[k]);
        }
    }
}

// Corrector (relaxingFluid.m:52-71): u*/2 and F* at cells -2 .. C+1 (index j + 2); ich = 1 / (2 c_f*), nh = -dt/dx c_f*.
// (Not on 2R and 2L: the limiter's product would underflow elsewhere.)  The limited fluxes' own const ghosts: the
// lower one copies cell 0's, the upper one that of end_k (the local cell at a const upper end, or C).
template <typename V, int C, int LIM>
__device__ __forceinline__ void seg_correct(const V (&u)[C], const V (&uh)[C + 4], const V (&Fs)[C + 4], V ich, V nich,
                                            V nh, bool lo_end, int end_k, V (&unew)[C]) {
    // R at cells j-1 .. j+1 and the difference below j (L likewise), rolled over j = -1 .. C
    V R1 = v_fma(Fs[1], ich, uh[1]), L1, Rp, Lp, dR = v_sub(R1, v_fma(Fs[0], ich, uh[0])), dL, a;
    L1 = v_fma(Fs[1], nich, uh[1]);
#pragma unroll
    for (int j = -1; j <= C; ++j) {
        V Rl, Ll;
        if (j < C) {
            const V R2 = v_fma(Fs[j + 3], ich, uh[j + 3]), d = v_sub(R2, R1);
            Rl = v_add(R1, v_limit<LIM>(dR, d));
            R1 = R2;
            dR = d;
        }
        {
            const V L2 = v_fma(Fs[j + 3], nich, uh[j + 3]), d = v_sub(L2, L1);
            if (j >= 0) Ll = v_sub(L1, v_limit<LIM>(dL, d));   // the limiters are odd
            L1 = L2;
            dL = d;
        }
        if (j >= 1) unew[j - 1] = v_fma(nh, v_sub(a, v_pick(j - 1 == end_k, Lp, Ll)), u[j - 1]);
        if (j >= 0 && j < C) {
            if (j == 0) Rp = v_pick(lo_end, Rl, Rp);
            a = v_add(v_sub(Rl, Rp), Ll);
        }
        Rp = Rl;
        Lp = Ll;
    }
}

// Values of variables v, v + 1 (or v alone) as one lane.
template <typename V, typename T> struct SegLane {
    static constexpr int N = 1;
    static __device__ __forceinline__ V get(T a, T) { return a; }
    static __device__ __forceinline__ void put(V x, T& a, T&) { a = x; }
};
template <> struct SegLane<F2, float> {
    static constexpr int N = 2;
    static __device__ __forceinline__ F2 get(float a, float b) { return F2(a, b); }
    static __device__ __forceinline__ void put(F2 x, float& a, float& b) { x.get(a, b); }
};

// Cell k (known at compile time) of the segment's variables.
template <typename T, int C>
__device__ __forceinline__ void cell(const T (&w)[5][C], int k, T (&c)[5]) {
#pragma unroll
    for (int v = 0; v < 5; ++v) c[v] = w[v][k];
}
// Whether cell k (known at compile time) is the n-th.  The comparison is kept opaque: seen together, a chain
// of them over k becomes one access at a run-time index, which would move the whole array out of registers.
__device__ __forceinline__ bool is_cell(int k, int n) {
    asm("" : "+r"(n));
    return k == n;
}
// What the stages need to know of a thread's place: its neighbours' records, the ends it sits at, its own cells.
struct SegEnds {
    unsigned round;          // seg_predict: the cells that round (bit k)
    SegRef l1, l2, r1, r2;   // cells -1, -2 and the two past the last own cell
    bool circ_lo, circ_hi;
    bool solo;               // the whole pencil in this thread: its neighbours are its own cells
    bool lo_own, hi_own;     // a const end below / above
    int nown, NT;
};

// Predictor of variables v .. (one lane's) in place: u becomes u*.
template <typename V, typename T, int C, int RND, int v>
__device__ __forceinline__ void seg_predict_vars(const SegEnds& e, T (&u)[5][C], const T (&F)[5][C], T ic, T qh) {
    using L = SegLane<V, T>;
    constexpr int M = L::N, w = v + M - 1;
    T ul[M], Fl[M], ur[M], Fr[M];
    if (e.solo) {
#pragma unroll
        for (int m = 0; m < M; ++m) {
            ul[m] = e.circ_lo ? u[v + m][C - 1] : u[v + m][0];
            Fl[m] = e.circ_lo ? F[v + m][C - 1] : F[v + m][0];
            ur[m] = e.circ_hi ? u[v + m][0] : u[v + m][C - 1];
            Fr[m] = e.circ_hi ? F[v + m][0] : F[v + m][C - 1];
        }
    } else {
        rec_part<v, M>(e.l1.X1, 2, e.l1.i1, e.NT, ul, Fl);
        rec_part<v, M>(e.r1.X1, 2, e.r1.i1, e.NT, ur, Fr);
    }
    V a[C + 2], f[C + 2], o[C];
    a[0] = L::get(ul[0], ul[M - 1]);
    f[0] = L::get(Fl[0], Fl[M - 1]);
    a[C + 1] = L::get(ur[0], ur[M - 1]);
    f[C + 1] = L::get(Fr[0], Fr[M - 1]);
#pragma unroll
    for (int k = 0; k < C; ++k) { a[k + 1] = L::get(u[v][k], u[w][k]); f[k + 1] = L::get(F[v][k], F[w][k]); }
    if (e.nown < C) {   // the cell past a ragged end
#pragma unroll
        for (int k = 1; k < C; ++k) {
            const bool here = is_cell(k, e.nown);
            a[k + 1] = v_pick(here, a[C + 1], a[k + 1]);
            f[k + 1] = v_pick(here, f[C + 1], f[k + 1]);
        }
    }
    seg_predict<V, C, v < 4 ? RND : 0>(a, f, v_dup<V>(ic), v_dup<V>(-ic), v_dup<V>(qh), v_dup<V>(-qh), e.round, o);
#pragma unroll
    for (int k = 0; k < C; ++k) L::put(o[k], u[v][k], u[w][k]);
}

// Corrector of variables v .. (one lane's): the new values of the own cells from u, u* and F*, stored
// at once (held to the end they would cost 5 C registers).
template <typename V, typename T, int C, int LIM, int v, typename Store>
__device__ __forceinline__ void seg_correct_vars(const SegEnds& e, const T (&u)[5][C], const Store& store,
                                                 const T (&us)[5][C], const T (&Fs)[5][C], T ics, T ffc) {
    using L = SegLane<V, T>;
    constexpr int M = L::N, w = v + M - 1;
    V x[C + 4], f[C + 4], o[C], a[C];
#pragma unroll
    for (int k = 0; k < C; ++k) {
        x[k + 2] = L::get(us[v][k], us[w][k]);
        f[k + 2] = L::get(Fs[v][k], Fs[w][k]);
    }
    if (e.solo) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {   // cells -2, -1 and C, C + 1
            x[j] = e.circ_lo ? x[C + j] : x[2];
            f[j] = e.circ_lo ? f[C + j] : f[2];
            x[C + 2 + j] = e.circ_hi ? x[2 + j] : x[C + 1];
            f[C + 2 + j] = e.circ_hi ? f[2 + j] : f[C + 1];
        }
    } else {
        T p[M], q[M];
        rec_part<v, M>(e.l2.X2, 4, e.l2.i2, e.NT, p, q);
        x[0] = L::get(p[0], p[M - 1]);
        f[0] = L::get(q[0], q[M - 1]);
        rec_part<v, M>(e.l1.X2, 4, e.l1.i2, e.NT, p, q);
        x[1] = L::get(p[0], p[M - 1]);
        f[1] = L::get(q[0], q[M - 1]);
        rec_part<v, M>(e.r1.X2, 4, e.r1.i2, e.NT, p, q);
        x[C + 2] = L::get(p[0], p[M - 1]);
        f[C + 2] = L::get(q[0], q[M - 1]);
        rec_part<v, M>(e.r2.X2, 4, e.r2.i2, e.NT, p, q);
        x[C + 3] = L::get(p[0], p[M - 1]);
        f[C + 3] = L::get(q[0], q[M - 1]);
    }
    if (e.nown < C) {   // the two cells past a ragged end: local cells nown and nown + 1
#pragma unroll
        for (int k = 1; k < C; ++k) {
            const bool one = is_cell(k, e.nown), two = is_cell(k, e.nown + 1);
            x[k + 2] = v_pick(one, x[C + 2], v_pick(two, x[C + 3], x[k + 2]));
            f[k + 2] = v_pick(one, f[C + 2], v_pick(two, f[C + 3], f[k + 2]));
        }
        const bool next = is_cell(C - 1, e.nown);
        x[C + 2] = v_pick(next, x[C + 3], x[C + 2]);
        f[C + 2] = v_pick(next, f[C + 3], f[C + 2]);
    }
#pragma unroll
    for (int k = 0; k < C; ++k) a[k] = L::get(u[v][k], u[w][k]);
#pragma unroll
    for (int j = 0; j < C + 4; ++j) x[j] = v_mul(x[j], v_splat<V>(0.5));
    seg_correct<V, C, LIM>(a, x, f, v_dup<V>(T(0.5) * ics), v_dup<V>(T(-0.5) * ics), v_dup<V>(-ffc), e.lo_own,
                           e.hi_own ? e.nown - 1 : C, o);
    T p[C], q[C];
#pragma unroll
    for (int k = 0; k < C; ++k) {
        if constexpr (M == 2) L::put(o[k], p[k], q[k]);
        else p[k] = o[k];
    }
    store(v, p);
    if constexpr (M == 2) store(w, q);
}

template <typename T, int C, int LIM, typename Store>
__device__ __forceinline__ void seg_correct_all(const SegEnds& e, const T (&u)[5][C], const Store& store,
                                                const T (&us)[5][C], const T (&Fs)[5][C], T ics, T ffc) {
    if constexpr (sizeof(T) == 4) {
        seg_correct_vars<F2, T, C, LIM, 0>(e, u, store, us, Fs, ics, ffc);
        asm volatile("" ::: "memory");   // one lane's neighbours at a time: fewer live registers
        seg_correct_vars<F2, T, C, LIM, 2>(e, u, store, us, Fs, ics, ffc);
        asm volatile("" ::: "memory");
        seg_correct_vars<T, T, C, LIM, 4>(e, u, store, us, Fs, ics, ffc);
    } else {
        seg_correct_vars<T, T, C, LIM, 0>(e, u, store, us, Fs, ics, ffc);
        seg_correct_vars<T, T, C, LIM, 1>(e, u, store, us, Fs, ics, ffc);
        seg_correct_vars<T, T, C, LIM, 2>(e, u, store, us, Fs, ics, ffc);
        seg_correct_vars<T, T, C, LIM, 3>(e, u, store, us, Fs, ics, ffc);
        seg_correct_vars<T, T, C, LIM, 4>(e, u, store, us, Fs, ics, ffc);
    }
}

// ---- fade ends (fade_shift.m:21-45) ---------------------------------------------------------------------
// The damping of one cell's row in a shifted array: v toward the shifted array's first value (s0, weight
// lo), then toward its last (sN, weight hi); weights are 0 (and nothing is done) away from the ends.  The share of v
// is rounded first, and in FP32 the half step's change too except the energy's, as in the pencil-tile kernels.
template <typename T>
struct SegFade {
    T lo, hi;
    __device__ __forceinline__ T operator()(T v, T s0, T sN) const {
        if (lo != T(0)) v = v_fma(lo, s0, (T(1) - lo) * v);
        if (hi != T(0)) v = v_fma(hi, sN, (T(1) - hi) * v);
        return v;
    }
};

// Publish the last two own cells of a segment of n < C cells: the last in slot b, the one before in slot a (n >= 2;
// a < 0: not published).  Every cell is written, those not wanted to slot 0, which the caller writes
// afterwards: the choice is in the address, since a choice among the cells' values (by selects or by branches)
// moves their arrays out of registers.
template <typename T, int C>
__device__ __forceinline__ void rec_put_tail(unsigned char* X, int slots, int a, int b, int NT, int t, const T (&u)[5][C],
                                             const T (&F)[5][C], int n) {
#pragma unroll
    for (int k = C - 2; k >= 0; --k) {
        T c[5], f[5];
        cell(u, k, c);
        cell(F, k, f);
        rec_put(X, slots, is_cell(k, n - 1) ? b : (a >= 0 && is_cell(k, n - 2) ? a : 0), NT, t, c, f);
    }
}

// VT: the artificial viscosity (VISC_*), fixed per kernel.  With viscosity each of the first two
// stages takes one more barrier: the viscosity exchange set is published with the pencil maximum, and
// the flux numerators (which include the viscous pressure) are published after it; every segment is whole.
// CLU: one pencil along x per cluster of CL CTAs (CL = 1: one CTA).  FADE: a fade end on this dimension.
template <typename T, int MHD, int C, int VT, bool CLU, bool FADE>
__device__ __forceinline__ void fluid_seg_body(const FluidArgs& a, unsigned vblock) {
    static_assert(!CLU || VT == VISC_NONE, "cluster segments carry no viscosity");
    static_assert(!FADE || (VT == VISC_NONE && !CLU), "fade ends: one CTA, no viscosity");
    static_assert(C >= 2, "two cells per end are published");
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double cflp[3][MAX_WARPS];
    using U = typename SegBits<T>::U;
    const SweepGeom& g = a.sg;
    // (a batch may launch a member's CTAs with more threads than its tiling has: they idle)
    const int NT = CLU ? g.NT : (int)blockDim.x, S = g.G, d = g.d, d1 = g.d1, d2 = g.d2, N = g.N;
    const int t = threadIdx.x;
    SegPos sp;
    sp.init<CLU>(g, vblock);
    const int s = sp.s, r0 = s * C;
    const int nown = sp.colok ? (N - r0 < C ? N - r0 : C) : 0;   // own cells inside the pencil (idle threads: none)
    unsigned char* X1 = smem;                            // (u, F) of the first and the last own cell
    unsigned char* X2 = X1 + 2 * seg_rec_bytes<T>() * NT;   // (u*, F*) of own cells 0, 1, last - 1, last
    U* pmax = reinterpret_cast<U*>(X2 + 4 * seg_rec_bytes<T>() * NT);   // [2][Wb] pencil maxima
    double* V = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(pmax) + 16 * g.Wb);   // viscosity or fade anchors
    for (int i = t; i < 2 * g.Wb; i += NT) pmax[i] = 0;

    // ---- the neighbour segments --------------------------------------------------------------------
    SegEnds e;
    const bool circ_lo = a.mode[CLS_MASS][0] == BC_CIRC, circ_hi = a.mode[CLS_MASS][1] == BC_CIRC;
    e.circ_lo = circ_lo;
    e.circ_hi = circ_hi;
    e.solo = VT == VISC_NONE && !CLU && !FADE && S == 1 && N == C;   // uniform over the launch
    e.nown = nown;
    e.NT = NT;
    const bool solo = e.solo;
    const int ls = d == 0 ? 1 : g.Wb;     // thread distance between consecutive segments of a pencil
    const bool lo_own = s == 0 && !circ_lo, hi_own = s == S - 1 && !circ_hi;
    e.lo_own = lo_own;
    const bool tile = sizeof(T) == 4 && a.round_cells == 0;
    e.round = 0;
    if (sizeof(T) == 4 && a.round_cells)
#pragma unroll
        for (int k = 0; k < C; ++k)
            if (C == 3 || k == C - 1 || k % 4 == 3) e.round |= (unsigned)((r0 + k + 1) % a.round_cells == 0) << k;
    e.hi_own = hi_own;
    SegRef &rl1 = e.l1, &rl2 = e.l2, &rr1 = e.r1, &rr2 = e.r2;
    int lt, rt;                  // threads of the neighbour segments (viscosity: whole segments, one CTA)
    {
        const int me = sp.colok ? s : (CLU ? S - 1 : 0);   // idle threads: the records of some segment
        const int last_n = N - (S - 1) * C;                 // own cells of the last segment
        const int sl = me > 0 ? me - 1 : (circ_lo ? S - 1 : 0);
        const int sr = me < S - 1 ? me + 1 : (circ_hi ? 0 : S - 1);
        const int sll = sl > 0 ? sl - 1 : (circ_lo ? S - 1 : 0);
        const int srr = sr < S - 1 ? sr + 1 : (circ_hi ? 0 : S - 1);
        // record of segment q: slot k1 of the first set, slot k2 of the second
        auto ref = [&](int q, int k1, int k2) -> SegRef {
            SegRef r;
            int tq;
            r.X1 = X1;
            r.X2 = X2;
            if constexpr (CLU) {
                const int rk = q / NT;
                tq = q - rk * NT;
                if (rk != sp.rank) {
                    r.X1 = cg::this_cluster().map_shared_rank(X1, rk);
                    r.X2 = cg::this_cluster().map_shared_rank(X2, rk);
                }
            } else {
                tq = sp.colok ? t + (q - s) * ls : t;
            }
            r.i1 = k1 * NT + tq;
            r.i2 = k2 * NT + tq;
            return r;
        };
        const bool lo_me = me == 0 && !circ_lo, hi_me = me == S - 1 && !circ_hi;
        // a const end's ghosts are its end cell: slot 0 of the first segment, the last slot of the last one
        rl1 = lo_me ? ref(me, 0, 0) : ref(sl, 1, 3);
        rr1 = hi_me ? ref(me, 1, 3) : ref(sr, 0, 0);
        const bool l_short = sl == S - 1 && last_n == 1, r_short = sr == S - 1 && last_n == 1;
        rl2 = lo_me ? rl1 : (l_short ? ref(sll, 1, 3) : ref(sl, 1, 2));
        rr2 = hi_me ? rr1 : (r_short ? (circ_hi ? ref(srr, 0, 0) : ref(sr, 1, 3)) : ref(sr, 0, 1));
        lt = s > 0 ? t - ls : (circ_lo ? t + (S - 1) * ls : t);
        rt = s < S - 1 ? t + ls : (circ_hi ? t - (S - 1) * ls : t);
    }

    // ---- stage 1: load, pressure, speed, F -----------------------------------------------------------
    // vector accesses need segments on multiples of C: pencils start on one where C divides N
    const bool vec = d == 0 && N % C == 0;
    const int sd = (int)g.sd;
    const int o0 = sp.base + r0 * sd;
    // momentum and cell-centred B in sweep-rotated order: component 0 along the sweep, then d1, d2
    void* const qv[5] = {a.q[Q_RHO], a.q[Q_PX + d], a.q[Q_PX + d1], a.q[Q_PX + d2], a.q[Q_E]};
    void* const bv[3] = {a.q[Q_CBX + d], a.q[Q_CBX + d1], a.q[Q_CBX + d2]};
    const bool ub[3] = {a.use_b[d] != 0, a.use_b[d1] != 0, a.use_b[d2] != 0};
    // rotated slots of the natural x, y, z components (the CSW sound speed sums in natural order)
    const int nx = d == 0 ? 0 : (d1 == 0 ? 1 : 2), ny = d == 1 ? 0 : (d1 == 1 ? 1 : 2), nz = d == 2 ? 0 : (d1 == 2 ? 1 : 2);
    constexpr bool LOADB = MHD || VT == VISC_CSW;   // cswSoundSpeed reads every cell-centred component
    pdl_wait();
    const int stop = a.tm->done | (!CLU || g.CL == 1 ? a.tm->error : a.tm->halt);   // (clusters: fluid_sweep_body_general)
    const double dtx = quotient_by(a.tm->dt, a.dx, a.inv_dx);
    T u[5][C], bb[3][C], F[5][C];
    auto load_u = [&](int v, T (&w)[C]) { win_load<T, C, true>(qv[v], o0, sd, vec, nown, v == 0 ? T(1) : T(0), w); };
    auto load_b = [&]() {   // the cell-centred B, which a fluid sweep leaves alone
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (LOADB) win_load<T, C, true>(bv[c], o0, sd, vec, nown, T(0), bb[c]);
            else
#pragma unroll
                for (int k = 0; k < C; ++k) bb[c][k] = T(0);
        }
    };
#pragma unroll
    for (int v = 0; v < 5; ++v) load_u(v, u[v]);
    load_b();
    SegFade<T> fw[C];
    const bool fade_lo = FADE && a.mode[CLS_MASS][0] == BC_FADE, fade_hi = FADE && a.mode[CLS_MASS][1] == BC_FADE;
    if constexpr (FADE) {
        const int f = a.fade_f;
#pragma unroll
        for (int k = 0; k < C; ++k) {
            const int r = r0 + k;
            fw[k].lo = k < nown && r < f ? (T)a.fade[r] : T(0);
            fw[k].hi = k < nown && r >= N - f ? (T)a.fade[N - 1 - r] : T(0);
        }
    }
    if (stop) return;   // after the loads are on their way: the flags take as long as they do
    __syncthreads();    // the maxima are zeroed
    T u0[5][C];   // the variables before the sweep
#pragma unroll
    for (int v = 0; v < 5; ++v)
#pragma unroll
        for (int k = 0; k < C; ++k) u0[v][k] = u[v][k];
    const SegPressure pk(a.gamma);
    // sum of squares of the cell-centred B components without isZero
    auto bsq = [&](int k) {
        double m = 0.0;
        if constexpr (MHD)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                if (ub[c]) m = fma((double)bb[c][k], (double)bb[c][k], m);
        return m;
    };
    const bool whole = nown == C;
    auto put1 = [&](const T (&w)[5][C], const T (&Fw)[5][C]) {
        if (solo) return;
        T c[5], f[5];
        if (!whole) {
            rec_put_tail(X1, 2, -1, 1, NT, t, w, Fw, nown);
        } else {
            cell(w, C - 1, c);
            cell(Fw, C - 1, f);
            rec_put(X1, 2, 1, NT, t, c, f);
        }
        cell(w, 0, c);
        cell(Fw, 0, f);
        rec_put(X1, 2, 0, NT, t, c, f);
    };
    // fade: (w, F) of the pencil's rows 0, 1, N-2, N-1 as anchor records of stage st
    T* AN = reinterpret_cast<T*>(V);
    const int ab = sp.b < g.Wb ? sp.b : 0;   // idle threads past the pencils read pencil 0's
    const bool near_end = r0 < 2 || r0 + C > N - 2;
    auto row_slot = [&](int r) { return r == 0 ? 0 : (r == 1 ? 1 : (r == N - 2 ? 2 : (r == N - 1 ? 3 : -1))); };
    auto put_anchors = [&](int st, const T (&w)[5][C], const T (&Fw)[5][C]) {
        if (!near_end) return;
#pragma unroll
        for (int k = 0; k < C; ++k) {
            const int q = k < nown ? row_slot(r0 + k) : -1;
            if (q >= 0) {
                T* p = AN + ((st * 4 + q) * g.Wb + sp.b) * 10;
#pragma unroll
                for (int v = 0; v < 5; ++v) { p[v] = w[v][k]; p[5 + v] = Fw[v][k]; }
            }
        }
    };
    T lmax = T(0), cf;
    if constexpr (VT == VISC_NONE) {
#pragma unroll
        for (int k = 0; k < C; ++k) {
            T c[5], Fk[5], p, cs, ir;
            cell(u, k, c);
            const T b3[3] = {bb[0][k], bb[1][k], bb[2][k]};
            const T spd = seg_pressure<MHD>(pk, c, bsq(k), p, cs, ir);
            if (k < nown) lmax = fmax(lmax, spd);
            seg_flux<T, MHD>(d, tile, c, b3, p, ir, Fk);
#pragma unroll
            for (int v = 0; v < 5; ++v) F[v][k] = Fk[v];
        }
        put1(u, F);
        if constexpr (FADE) put_anchors(0, u, F);
        seg_max_publish<T, CLU>(g, sp, lmax, pmax);
        if (!solo) sp_sync<CLU>(g);
        cf = seg_max_collect<T, CLU>(g, sp, lmax, pmax);   // freezing speed (wFluidFlux.m:18-22)
    } else {
        T P[C], CS[C], IR[C];
        double vel[C], snd[C], q[C];
#pragma unroll
        for (int k = 0; k < C; ++k) {
            T c[5];
            cell(u, k, c);
            const T spd = seg_pressure<MHD>(pk, c, bsq(k), P[k], CS[k], IR[k]);
            if (k < nown) lmax = fmax(lmax, spd);
        }
        seg_visc_publish<T, C, VT>(u, bb, a.gamma, nx, ny, nz, V, NT, t, vel, snd);
        seg_max_publish<T, CLU>(g, sp, lmax, pmax);
        __syncthreads();
        cf = seg_max_collect<T, CLU>(g, sp, lmax, pmax);   // freezing speed (wFluidFlux.m:18-22), before the viscosity
        seg_visc_terms<T, C, VT>(a, a.gamma, u, CS, vel, snd, V, NT, lt, rt, lo_own, hi_own, q);
#pragma unroll
        for (int k = 0; k < C; ++k) {
            T c[5], Fk[5];
            cell(u, k, c);
            const T b3[3] = {bb[0][k], bb[1][k], bb[2][k]};
            seg_flux<T, MHD>(d, tile, c, b3, visc_add<T>(P[k], q[k]), IR[k], Fk);   // press + viscosity.solve (wFluidFlux.m:24)
#pragma unroll
            for (int v = 0; v < 5; ++v) F[v][k] = Fk[v];
        }
        put1(u, F);
        __syncthreads();
    }

    // ---- stage 2: predictor (relaxingFluid.m:30-39) and the half-step pressure, speed, F ----------
    T ic;
    if constexpr (sizeof(T) == 4) ic = __frcp_rn(cf);
    else ic = recip(cf);
    const T hfc = (T)(0.5 * dtx) * cf;
    if constexpr (!FADE) {
        const T qh = T(0.5) * hfc;
        constexpr int RND = seg_round_mode<T, MHD, C>();
        if constexpr (sizeof(T) == 4) {
            seg_predict_vars<F2, T, C, RND, 0>(e, u, F, ic, qh);
            asm volatile("" ::: "memory");   // one lane's neighbours at a time: fewer live registers
            seg_predict_vars<F2, T, C, RND, 2>(e, u, F, ic, qh);
            asm volatile("" ::: "memory");
            seg_predict_vars<T, T, C, RND, 4>(e, u, F, ic, qh);
        } else {
            seg_predict_vars<T, T, C, RND, 0>(e, u, F, ic, qh);
            seg_predict_vars<T, T, C, RND, 1>(e, u, F, ic, qh);
            seg_predict_vars<T, T, C, RND, 2>(e, u, F, ic, qh);
            seg_predict_vars<T, T, C, RND, 3>(e, u, F, ic, qh);
            seg_predict_vars<T, T, C, RND, 4>(e, u, F, ic, qh);
        }
    } else {
        T ul[5], Fl[5], ur[5], Fr[5];
        rec_get(rl1.X1, 2, rl1.i1, NT, ul, Fl);
        rec_get(rr1.X1, 2, rr1.i1, NT, ur, Fr);
        const T* an = AN + ab * 10;
        const int ar = 10 * g.Wb;   // between anchor rows
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            T R[C + 1], L[C + 1];   // R at cells -1 .. C-1 (j + 1), L at cells 0 .. C (j)
            R[0] = T(0.5) * v_fma(Fl[v], ic, ul[v]);
            L[C] = T(0.5) * v_fma(Fr[v], -ic, ur[v]);
#pragma unroll
            for (int k = 0; k < C; ++k) {
                R[k + 1] = T(0.5) * v_fma(F[v][k], ic, u[v][k]);
                L[k] = T(0.5) * v_fma(F[v][k], -ic, u[v][k]);
            }
            const T Le = L[C];   // past a ragged end
#pragma unroll
            for (int k = 1; k < C; ++k) L[k] = v_pick(is_cell(k, nown), Le, L[k]);
            const T R0 = T(0.5) * v_fma(an[5 + v], ic, an[v]), RN = T(0.5) * v_fma(an[2 * ar + 5 + v], ic, an[2 * ar + v]);
            const T L0 = T(0.5) * v_fma(an[ar + 5 + v], -ic, an[ar + v]), LN = T(0.5) * v_fma(an[3 * ar + 5 + v], -ic, an[3 * ar + v]);
#pragma unroll
            for (int k = 0; k < C; ++k) {
                const T Rm = fade_lo ? fw[k](R[k], R0, RN) : R[k], Lp = fade_hi ? fw[k](L[k + 1], L0, LN) : L[k + 1];
                const T change = R[k + 1] - Rm + L[k] - Lp;
                u[v][k] = sizeof(T) == 4 && v < 4 ? u[v][k] - hfc * change : v_fma(-hfc, change, u[v][k]);
            }
        }
    }
    T (&us)[5][C] = u, Fs[5][C];   // the half-step state in u's place
    T lmax2 = T(0), cfs;
    const T mm = (T)a.minmass;
    {
        T P2[C], CS2[C], IR2[C];
#pragma unroll
        for (int k = 0; k < C; ++k) {
            us[0][k] = us[0][k] > mm ? us[0][k] : mm;   // max(rho, MINMASS), NaN -> MINMASS
            if (k >= nown) { us[0][k] = T(1); us[1][k] = us[2][k] = us[3][k] = us[4][k] = T(0); }
            T c[5], Fk[5];
            cell(us, k, c);
            const T spd = seg_pressure<MHD>(pk, c, bsq(k), P2[k], CS2[k], IR2[k]);   // relaxingFluid.m:47-50
            if (k < nown) lmax2 = fmax(lmax2, spd);
            if constexpr (VT == VISC_NONE) {
                const T b3[3] = {bb[0][k], bb[1][k], bb[2][k]};
                seg_flux<T, MHD>(d, tile, c, b3, P2[k], IR2[k], Fk);
#pragma unroll
                for (int v = 0; v < 5; ++v) Fs[v][k] = Fk[v];
            }
        }
        if constexpr (VT != VISC_NONE) {
            // the viscosity of the half-step state: one more barrier before its fluxes are published
            double vel[C], snd[C], q[C];
            seg_visc_publish<T, C, VT>(us, bb, a.gamma, nx, ny, nz, V, NT, t, vel, snd);
            seg_max_publish<T, CLU>(g, sp, lmax2, pmax + g.Wb);
            __syncthreads();
            seg_visc_terms<T, C, VT>(a, a.gamma, us, CS2, vel, snd, V, NT, lt, rt, lo_own, hi_own, q);
#pragma unroll
            for (int k = 0; k < C; ++k) {
                T c[5], Fk[5];
                cell(us, k, c);
                const T b3[3] = {bb[0][k], bb[1][k], bb[2][k]};
                seg_flux<T, MHD>(d, tile, c, b3, visc_add<T>(P2[k], q[k]), IR2[k], Fk);
#pragma unroll
                for (int v = 0; v < 5; ++v) Fs[v][k] = Fk[v];
            }
        }
    }
    if (!solo) {
        T c[5], f[5];
        if (!whole) {
            rec_put_tail(X2, 4, 2, 3, NT, t, us, Fs, nown);
        } else {
            cell(us, C - 2, c);
            cell(Fs, C - 2, f);
            rec_put(X2, 4, 2, NT, t, c, f);
            cell(us, C - 1, c);
            cell(Fs, C - 1, f);
            rec_put(X2, 4, 3, NT, t, c, f);
        }
        cell(us, 0, c);
        cell(Fs, 0, f);
        rec_put(X2, 4, 0, NT, t, c, f);
        cell(us, 1, c);
        cell(Fs, 1, f);
        rec_put(X2, 4, 1, NT, t, c, f);
    }
    if constexpr (FADE) put_anchors(1, us, Fs);
    if constexpr (VT == VISC_NONE) seg_max_publish<T, CLU>(g, sp, lmax2, pmax + g.Wb);
    if (!solo) sp_sync<CLU>(g);
    cfs = seg_max_collect<T, CLU>(g, sp, lmax2, pmax + g.Wb);   // freezing speed of the half step
    T ics;
    if constexpr (sizeof(T) == 4) ics = __frcp_rn(cfs);
    else ics = recip(cfs);

    pdl_trigger();
    // ---- stage 3: corrector fluxes, TVD limiter, update (relaxingFluid.m:52-71) -------------------
    // each variable is stored as soon as it is updated: nobody else reads this thread's cells
    const T mo = (T)a.minmass_out;
    auto store_u = [&](int v, T (&w)[C]) {
        if (v == 0)
#pragma unroll
            for (int k = 0; k < C; ++k) w[k] = w[k] > mo ? w[k] : mo;
        win_store<T, C>(qv[v], o0, sd, vec, nown, w);
    };
    const T ffc = (T)dtx * cfs;
    if constexpr (!FADE) {
        if (a.limiter == LIM_VANLEER) seg_correct_all<T, C, LIM_VANLEER>(e, u0, store_u, us, Fs, ics, ffc);
        else if (a.limiter == LIM_SUPERBEE) seg_correct_all<T, C, LIM_SUPERBEE>(e, u0, store_u, us, Fs, ics, ffc);
        else seg_correct_all<T, C, LIM_MINMOD>(e, u0, store_u, us, Fs, ics, ffc);
    } else {
        T hl[5], hFl[5], hr[5], hFr[5];   // cell -1 and the one past the last own cell
        rec_get(rl1.X2, 4, rl1.i2, NT, hl, hFl);
        rec_get(rr1.X2, 4, rr1.i2, NT, hr, hFr);
        const T* an = AN + (4 * g.Wb + ab) * 10;
        const int ar = 10 * g.Wb;
        T Rl[5][C], Ll[5][C], e1[5], e2[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            T R[C + 2], L[C + 2];   // cells -1 .. C (j + 1)
#pragma unroll
            for (int j = -1; j <= C; ++j) {
                const bool past = j > 0 && j < C && is_cell(j, nown);   // past a ragged end
                const T x = j < 0 ? hl[v] : (j < C ? v_pick(past, hr[v], us[v][j < C && j >= 0 ? j : 0]) : hr[v]);
                const T f = j < 0 ? hFl[v] : (j < C ? v_pick(past, hFr[v], Fs[v][j < C && j >= 0 ? j : 0]) : hFr[v]);
                R[j + 1] = T(0.5) * v_fma(f, ics, x);
                L[j + 1] = T(0.5) * v_fma(f, -ics, x);
            }
            T aR[4], aL[4];   // rows 0, 1, N-2, N-1
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const T x = an[q * ar + v], f = an[q * ar + 5 + v];
                aR[q] = T(0.5) * v_fma(f, ics, x);
                aL[q] = T(0.5) * v_fma(f, -ics, x);
            }
#pragma unroll
            for (int k = 0; k < C; ++k) {
                const T r = R[k + 1], l = L[k + 1];
                const T Rm = fade_lo ? fw[k](R[k], aR[0], aR[2]) : R[k], Rp = fade_hi ? fw[k](R[k + 2], aR[1], aR[3]) : R[k + 2];
                const T Lm = fade_lo ? fw[k](L[k], aL[0], aL[2]) : L[k], Lp = fade_hi ? fw[k](L[k + 2], aL[1], aL[3]) : L[k + 2];
                T cr, cl;
                if (a.limiter == LIM_VANLEER) { cr = v_limit<LIM_VANLEER>(r - Rm, Rp - r); cl = v_limit<LIM_VANLEER>(Lm - l, l - Lp); }
                else if (a.limiter == LIM_SUPERBEE) { cr = v_limit<LIM_SUPERBEE>(r - Rm, Rp - r); cl = v_limit<LIM_SUPERBEE>(Lm - l, l - Lp); }
                else { cr = v_limit<LIM_MINMOD>(r - Rm, Rp - r); cl = v_limit<LIM_MINMOD>(Lm - l, l - Lp); }
                Rl[v][k] = r + cr;
                Ll[v][k] = l + cl;
            }
        }
        // the limited fluxes next to the segment and at the anchor rows (the first exchange set is free again)
        if (!whole) {
            rec_put_tail(X1, 2, -1, 1, NT, t, Rl, Ll, nown);
        } else {
            cell(Rl, C - 1, e1);
            cell(Ll, C - 1, e2);
            rec_put(X1, 2, 1, NT, t, e1, e2);
        }
        cell(Rl, 0, e1);
        cell(Ll, 0, e2);
        rec_put(X1, 2, 0, NT, t, e1, e2);
        T* lf = AN + 80 * g.Wb;   // [4][Wb][5]: Rl at rows 0 and N-2, Ll at rows 1 and N-1
        if (near_end) {
#pragma unroll
            for (int k = 0; k < C; ++k) {
                const int q = k < nown ? row_slot(r0 + k) : -1;
                if (q >= 0)
#pragma unroll
                    for (int v = 0; v < 5; ++v) lf[(q * g.Wb + sp.b) * 5 + v] = (q & 1) ? Ll[v][k] : Rl[v][k];
            }
        }
        __syncthreads();
        T Rn[5], Ln[5], x[5];   // Rl of cell -1, Ll past the last own cell
        rec_get(X1, 2, rl1.i1, NT, Rn, x);   // slot 1 of the left neighbour (a const end's is not used)
        rec_get(X1, 2, rr1.i1, NT, x, Ln);   // slot 0 of the right one
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            const int fr = 5 * g.Wb;
            T un[C];
            const T R0 = lf[ab * 5 + v], L0 = lf[fr + ab * 5 + v], RN = lf[2 * fr + ab * 5 + v], LN = lf[3 * fr + ab * 5 + v];
#pragma unroll
            for (int k = 0; k < C; ++k) {
                T Rm = k > 0 ? Rl[v][k > 0 ? k - 1 : 0] : (lo_own ? Rl[v][0] : Rn[v]);
                T Lp = k < C - 1 ? Ll[v][k < C - 1 ? k + 1 : 0] : Ln[v];
                if (k == nown - 1) Lp = hi_own ? Ll[v][k] : Ln[v];
                if (fade_lo) Rm = fw[k](Rm, R0, RN);
                if (fade_hi) Lp = fw[k](Lp, L0, LN);
                un[k] = v_fma(-ffc, Rl[v][k] - Rm + Ll[v][k] - Lp, u0[v][k]);
            }
            store_u(v, un);
        }
    }
    // the other ranks have read this CTA's exchange sets before it moves on (and may exit)
    if (CLU && g.CL > 1) cluster_sync();
    if (a.cfl) {   // fused CFL maxima of the new state, read back (TimeManager.m:65-77)
        double m3[3] = {0.0, 0.0, 0.0};   // rotated order
        bool bad = false;
#pragma unroll
        for (int v = 0; v < 5; ++v) load_u(v, u[v]);
#pragma unroll
        for (int k = 0; k < C; ++k)
            if (k < nown) {
                double sp3[3];
                cfl_speeds(a.gamma, (double)u[0][k], (double)u[1][k], (double)u[2][k], (double)u[3][k], (double)u[4][k], bsq(k), sp3);
                bad = bad || !isfinite(sp3[0] + sp3[1] + sp3[2]);
#pragma unroll
                for (int c = 0; c < 3; ++c) m3[c] = fmax(m3[c], sp3[c]);
            }
        if (a.cfl & CFL_CHECK_NONFINITE) flag_nonfinite(a.tm, bad);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            m3[c] = warp_max_nonneg(m3[c]);
            if (lane == 0) cflp[c][warp] = m3[c];
        }
        __syncthreads();
        if (threadIdx.x < 3) {   // one global atomic per CTA and direction (rotated slot of direction t)
            const int rc = threadIdx.x == d ? 0 : (threadIdx.x == d1 ? 1 : 2);
            double m = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, cflp[rc][w]);
            atomic_max_nonneg(&a.tm->maxbits[threadIdx.x], m);
        }
    }
}

// What bounds it (256^3 mixed, x, 343 us): warp issue -- the FP64 pressure recovery, the limiters and the fluxes --
// beside HBM, whose 872 MB need 135 us at the measured 6.46 TB/s; y and z (523 and 553 us) also wait for their strided
// rows of 32 bytes.  One FP32 lane per instruction and whole-CTA barriers around idle threads make that 408, 583 and
// 584 us.  FP64 and fade ends against the pencil tiles: 96^3 FP64 57, 66 and 66 us against 72, 112 and 106; 96^3
// hydrodynamic with fade ends, mixed, 50, 52 and 52 us against 77, 103 and 103.  At 128 registers 16 warps share an SM;
// 80 registers for 24 warps spill more than they hide (256^3 y 649 -> 704 us), and persistent CTAs that fetch the next
// bundle with cp.async lose to plain loads (x 345 -> 410 us, y 593 -> 1020 us: 4-byte copies of strided rows).
// FP64 kernels of 3 and 4 cells a thread take CTAs of at most 256 threads with all 255 registers a thread can
// have (MAXT): at 128 they spill.  The others run at 128, 16 warps an SM; FP64 CTAs above 256 threads spill and are still
// faster than the pencil tiles (y fluid sweep of 700^2: 70 us against 127, of 600^2: 61 against 107).
template <typename T, int MHD, int C, int VT, bool CLU, bool FADE, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) fluid_seg_kernel(const __grid_constant__ FluidArgs a) {
    fluid_seg_body<T, MHD, C, VT, CLU, FADE>(a, blockIdx.x);
}

template <typename T, int MHD, int C, bool CLU, bool FADE, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) fluid_seg_batch_kernel(const FluidArgs* __restrict__ args,
                                                                  const BlockMap* __restrict__ map) {
    __shared__ FluidArgs sa;
    const BlockMap bm = map[blockIdx.x];
    load_member_args(sa, args + bm.member);
    __syncthreads();
    fluid_seg_body<T, MHD, C, VISC_NONE, CLU, FADE>(sa, (unsigned)bm.block);
}

}  // namespace img
