// Window form of the magnet sweep along X (magnet/magnetFlux.m:14-31, magnet/relaxingMagnet.m:15-60,
// magnet/MagnetArray.m:36-38) for pencils with circ or const ends.
//
// Each thread owns C consecutive cells of a pencil and computes the upwind/TVD chain for them in registers;
// what its stencil needs of the neighbour segments it gets through shared memory: the corner velocity and B_I
// of two cells on each side, then, once computed, wMag of two cells on each side.
//   chain  per transverse component I: vg from rho, p_X at the pencil and its I-1 neighbour, the
//          1-2-1 smoothing, velocityFlow, store.fluxR, store, wMag, flux with the limiter; B_I updated
//          in place and the limited flux F_I written to scratch for the CT pass.
//   CT     C_I = F_I - F_I.shift(I,+1), D_I = C_I.shift(X,-1), B_X = (B_X - dt/dI1 D_1) - dt/dI2 D_2
//          in place, and the cell-centred B_X and B_I2.
// Pencil ends along X (mag-class BC): circ wraps; const makes every shifted array take its own end value
// (constant_shift.m), so after each stage the cells beyond the pencil's end copy the stage's value at the
// end cell.  Transverse shifts (along I) use circ or const too; other boundaries and stored-edge capture
// take the tile kernels (magnet_sweep.cuh), with the same arithmetic per cell up to round-off.
// A pencil's length need not be a multiple of C (the last segment is ragged: S = ceil(N / C) segments,
// threads past them idle), and along x a pencil longer than one CTA's segments spans the CTAs of a
// thread-block cluster (one pencil per cluster; segment s = rank * NT + thread), whose barriers then
// order the exchanges through DSMEM.  A pencil of C cells is one thread's and exchanges nothing.
#pragma once

#include "seg_fluid.cuh"

namespace img {

// Offset of the transverse neighbour pencil at I-1 (n = -1) or I+1 (n = +1) along component q's dimension for
// a pencil whose coordinate along it is ie, under a circ or const BC on that side; 0 means the pencil
// itself (const edge, or a dimension that is not shifted).
__device__ __forceinline__ int trans_offset(const MagArgs& a, int q, int ie, int n, int mode) {
    const int ne = a.nI[q], se = a.sI[q];
    const int wrap = mode == BC_CIRC ? (ne - 1) * se : 0;
    int o = n < 0 ? (ie > 0 ? -se : wrap) : (ie < ne - 1 ? se : -wrap);
    return a.shiftI[q] ? o : 0;
}

// Global row of window cell j of segment s (rows r0 + j, wrapped for circ, clamped for const ends).
// The window reaches 2 rows past a segment, so on a pencil shorter than that a row wraps more than once (the loops run
// at most a few times).
__host__ __device__ __forceinline__ int win_row_multi(int r, int N, bool circ_lo, bool circ_hi) {
    if (r < 0) {
        if (!circ_lo) return 0;
        do r += N; while (r < 0);
        return r;
    }
    if (r >= N) {
        if (!circ_hi) return N - 1;
        do r -= N; while (r >= N);
        return r;
    }
    return r;
}

// The same where one wrap suffices: rows r >= -N and r < 2N (a window that reaches H rows past its
// segment, on a pencil of N >= C + H rows: the last segment starts at row N - 1 at most).  Selects
// only, no loop; a host-side check of the looping form (the kernels look such rows up rarely enough for the loop).
__host__ __device__ __forceinline__ int win_row_once(int r, int N, bool circ_lo, bool circ_hi) {
    const int lo = circ_lo ? r + N : 0, hi = circ_hi ? r - N : N - 1;
    return r < 0 ? lo : (r >= N ? hi : r);
}

// Const ends: the window cells of a stage array A (local cells LO .. HI-1 at A[j + OFS]) past the
// pencil's lower end copy its row 0 (local cell lend = -r0), those past its upper end its last row
// (local cell hend = N - 1 - r0): the const ghost of every shifted array (constant_shift.m).  The stages
// reach 2 cells past a segment, so near an end several segments' windows cross it, and the end row
// may be a window cell rather than an own one (short segments, a ragged last segment).
template <typename T, int OFS, int LO, int HI>
__device__ __forceinline__ void const_fill(T* A, bool circ_lo, bool circ_hi, int lend, int hend) {
    if (!circ_lo && lend > LO) {
        T e = A[LO + OFS];
#pragma unroll
        for (int j = LO + 1; j < HI; ++j)
            if (j == lend) e = A[j + OFS];
#pragma unroll
        for (int j = LO; j < HI; ++j)
            if (j < lend) A[j + OFS] = e;
    }
    if (!circ_hi && hend < HI - 1) {
        T e = A[LO + OFS];
#pragma unroll
        for (int j = LO + 1; j < HI; ++j)
            if (j == hend) e = A[j + OFS];
#pragma unroll
        for (int j = LO; j < HI; ++j)
            if (j > hend) A[j + OFS] = e;
    }
}

// The segment placement of seg_fluid.cuh plus the pencil's coordinates along the transverse dims; G is
// the pencil's segment count S, over the CL CTAs of a cluster where CL > 1.  Offsets are 32-bit (grids
// have fewer than 2^31 cells): one multiply-add forms an address.
struct WinPos {
    int b, s, c1, c2;
    bool colok;
    int base;
    __device__ __forceinline__ void init(const SweepGeom& g, unsigned vblock) {
        int t = threadIdx.x;
        unsigned blk = vblock;
        if (g.CL > 1) {   // cluster rank r holds segments r * NT .. r * NT + NT - 1 of the bundle's pencil
            blk = g.div_cl.div(vblock);
            t += (int)(vblock - blk * (unsigned)g.CL) * g.NT;
        }
        const unsigned q = g.div_lanes.div((unsigned)t);
        if (g.d == 0) { b = (int)q; s = t - b * g.G; }
        else { s = (int)q; b = t - s * g.Wb; }
        const int col = (int)(blk * (unsigned)g.Wb + (unsigned)b);
        colok = col < (int)g.ncol && b < g.Wb && s < g.G;   // threads past the last segment idle
        const unsigned c = colok ? (unsigned)col : 0u;
        c2 = (int)g.div_n1.div(c);
        c1 = (int)(c - (unsigned)c2 * (unsigned)g.n1);
        base = c1 * (int)g.s1 + c2 * (int)g.s2;
    }
};

// Every read of the pencil's arrays before any in-place write: the CTA's barrier, or the cluster's.
__device__ __forceinline__ void win_barrier(const SweepGeom& g) {
    if (g.CL > 1) cluster_sync();
    else __syncthreads();
}

// ---- lanes of the chain: both transverse components at once (mixed form) or one at a time (FP64) ------
// The two components of a cell run the same arithmetic on their own numbers, so the mixed form carries them
// as one packed pair of FP32; FP64 takes the components one after the other.
template <typename T> struct ChainLane { using V = double; static constexpr int PASSES = 2; };
template <> struct ChainLane<float> { using V = F2; static constexpr int PASSES = 1; };
// 1 where x < 0, else 0 (also for NaN)
__device__ __forceinline__ F2 v_negative(F2 x) {
    float a, b;
    x.get(a, b);
    float m, n;
    asm("set.lt.f32.f32 %0, %1, 0f00000000;" : "=f"(m) : "f"(a));
    asm("set.lt.f32.f32 %0, %1, 0f00000000;" : "=f"(n) : "f"(b));
    return F2(m, n);
}
__device__ __forceinline__ double v_negative(double x) { return x < 0.0 ? 1.0 : 0.0; }

// One cell of the first exchange set: the corner velocity and B_I of a lane (both components in the mixed
// form).  The second set holds wMag of the lane.
template <typename V>
struct __align__(16) ChainRec {
    V vg, b;
};

template <typename T>
__host__ __device__ inline size_t chain_win_smem_bytes(int NT, int C) {
    return (size_t)ChainLane<T>::PASSES * 24 * NT * C;
}

// The upwind/TVD chain of one lane over a segment (magnetFlux.m:18-19, relaxingMagnet.m:17-51) in two parts,
// with the exchange of wMag between them.  First part: vr the corner velocity at cells -2 .. C+1 (index j + 2),
// b B_I at cells -1 .. C (j + 1); out: wMag at the own cells and velocityFlow at cells -1 .. C-1 (j + 1).
// FILL: a const end may be near: after each stage the cells past it take the end cell's value (const_fill).
template <typename V, int C, bool FILL>
__device__ __forceinline__ void chain_predict(const V (&vr)[C + 4], const V (&b)[C + 2], V ff, bool circ_lo, bool circ_hi,
                                              int lend, int hend, V (&Wm)[C], V (&vf)[C + 1]) {
    const V one = v_splat<V>(1.0), mone = v_splat<V>(-1.0), two = v_splat<V>(2.0), quarter = v_splat<V>(0.25);
    const V mff = v_mul(mone, ff);
    // vg = 0.25*(vg.shift(X,-1) + vg.shift(X,1) + 2*vg) and F = B_I * vg at cells -1 .. C
    V vg[C + 2], Fr[C + 2], fR[C + 1];
#pragma unroll
    for (int j = 0; j < C + 2; ++j) vg[j] = v_mul(quarter, v_fma(two, vr[j + 1], v_add(vr[j], vr[j + 2])));
    if constexpr (FILL) const_fill<V, 1, -1, C + 1>(vg, circ_lo, circ_hi, lend, hend);
#pragma unroll
    for (int j = 0; j < C + 2; ++j) Fr[j] = v_mul(b[j], vg[j]);
    if constexpr (FILL) const_fill<V, 1, -1, C + 1>(Fr, circ_lo, circ_hi, lend, hend);
    // velocityFlow = (vg + vg.shift(X,1)) < 0, store.fluxR = F*(1-vf) + F.shift(X,1)*vf (relaxingMagnet.m:17-24)
#pragma unroll
    for (int j = 0; j < C + 1; ++j) {
        vf[j] = v_negative(v_add(vg[j], vg[j + 1]));
        fR[j] = v_fma(Fr[j], v_fma(mone, vf[j], one), v_mul(Fr[j + 1], vf[j]));
    }
    if constexpr (FILL) const_fill<V, 1, -1, C>(vf, circ_lo, circ_hi, lend, hend);
    if constexpr (FILL) const_fill<V, 1, -1, C>(fR, circ_lo, circ_hi, lend, hend);
    // store = B_I - ff*(fluxR - fluxR.shift(X,-1)); wMag = store.*velGrid
#pragma unroll
    for (int k = 0; k < C; ++k) Wm[k] = v_mul(v_fma(mff, v_sub(fR[k + 1], fR[k]), b[k + 1]), vg[k + 1]);
}

// Second part: Wm at cells -2 .. C+1 (j + 2), vf at cells -1 .. C-1 (j + 1), b B_I at the own cells; out: the
// updated B_I and the limited flux.
template <typename V, int C, int LIM>
__device__ __forceinline__ void chain_correct(const V (&Wm)[C + 4], const V (&vf)[C + 1], const V (&b)[C], V ff,
                                              bool lo_end, V (&bnew)[C], V (&flux)[C]) {
    const V one = v_splat<V>(1.0), mone = v_splat<V>(-1.0);
    const V mff2 = v_mul(v_splat<V>(-2.0), ff);
    // flux and its TVD correction (relaxingMagnet.m:32-51) at cells -1 .. C-1 (j + 1)
    V Fl[C + 1];
#pragma unroll
    for (int j = 0; j <= C; ++j) {
        const V m1 = Wm[j], w = Wm[j + 1], p1 = Wm[j + 2], p2 = Wm[j + 3 < C + 4 ? j + 3 : j], v = vf[j];
        const V nv = v_fma(mone, v, one);
        const V fx = v_fma(w, nv, v_mul(p1, v));
        const V dR = v_sub(p1, v_fma(v, p2, v_mul(nv, w)));
        const V dL = v_sub(w, v_fma(v, p1, v_mul(nv, m1)));
        Fl[j] = v_add(fx, v_limit<LIM>(dL, dR));
    }
    if (lo_end) Fl[0] = Fl[1];   // the flux's own const ghost
    // B_I = B_I - 2ff*(flux - flux.shift(X,-1)) (relaxingMagnet.m:49)
#pragma unroll
    for (int k = 0; k < C; ++k) {
        bnew[k] = v_fma(mff2, v_sub(Fl[k + 1], Fl[k]), b[k]);
        flux[k] = Fl[k + 1];
    }
}

// The same for a pencil of C cells held whole by one thread: every stage has C cells, and a neighbour
// past an end is the other end's cell (circ) or the end cell (const).
template <typename V, int C, int LIM>
__device__ __forceinline__ void chain_whole(const V (&vr)[C], const V (&b)[C], V ff, bool circ_lo, bool circ_hi,
                                            V (&bnew)[C], V (&flux)[C]) {
    static_assert(C >= 2, "a shift by 2 wraps once");
    const V one = v_splat<V>(1.0), mone = v_splat<V>(-1.0), two = v_splat<V>(2.0), quarter = v_splat<V>(0.25);
    const V mff = v_mul(mone, ff), mff2 = v_mul(two, mff);
    auto at = [&](const V (&A)[C], int k) -> V {   // k is a constant after unrolling
        if (k < 0) return circ_lo ? A[(k + C) % C] : A[0];
        if (k >= C) return circ_hi ? A[k % C] : A[C - 1];
        return A[k];
    };
    V vg[C], Fr[C], vf[C], fR[C], Wm[C], Fl[C];
#pragma unroll
    for (int k = 0; k < C; ++k) vg[k] = v_mul(quarter, v_fma(two, vr[k], v_add(at(vr, k - 1), at(vr, k + 1))));
#pragma unroll
    for (int k = 0; k < C; ++k) Fr[k] = v_mul(b[k], vg[k]);
#pragma unroll
    for (int k = 0; k < C; ++k) {
        vf[k] = v_negative(v_add(vg[k], at(vg, k + 1)));
        fR[k] = v_fma(Fr[k], v_fma(mone, vf[k], one), v_mul(at(Fr, k + 1), vf[k]));
    }
#pragma unroll
    for (int k = 0; k < C; ++k) Wm[k] = v_mul(v_fma(mff, v_sub(fR[k], at(fR, k - 1)), b[k]), vg[k]);
#pragma unroll
    for (int k = 0; k < C; ++k) {
        const V m1 = at(Wm, k - 1), w = Wm[k], p1 = at(Wm, k + 1), p2 = at(Wm, k + 2), v = vf[k];
        const V nv = v_fma(mone, v, one);
        const V fx = v_fma(w, nv, v_mul(p1, v));
        const V dR = v_sub(p1, v_fma(v, p2, v_mul(nv, w)));
        const V dL = v_sub(w, v_fma(v, p1, v_mul(nv, m1)));
        Fl[k] = v_add(fx, v_limit<LIM>(dL, dR));
    }
#pragma unroll
    for (int k = 0; k < C; ++k) {
        bnew[k] = v_fma(mff2, v_sub(Fl[k], at(Fl, k - 1)), b[k]);
        flux[k] = Fl[k];
    }
}

template <typename V, int C>
__device__ __forceinline__ void chain_correct_lim(int lim, const V (&Wm)[C + 4], const V (&vf)[C + 1], const V (&b)[C], V ff,
                                                  bool lo_end, V (&bnew)[C], V (&flux)[C]) {
    if (lim == LIM_VANLEER) chain_correct<V, C, LIM_VANLEER>(Wm, vf, b, ff, lo_end, bnew, flux);
    else if (lim == LIM_SUPERBEE) chain_correct<V, C, LIM_SUPERBEE>(Wm, vf, b, ff, lo_end, bnew, flux);
    else chain_correct<V, C, LIM_MINMOD>(Wm, vf, b, ff, lo_end, bnew, flux);
}
template <typename V, int C>
__device__ __forceinline__ void chain_whole_lim(int lim, const V (&vr)[C], const V (&b)[C], V ff, bool circ_lo,
                                                bool circ_hi, V (&bnew)[C], V (&flux)[C]) {
    if (lim == LIM_VANLEER) chain_whole<V, C, LIM_VANLEER>(vr, b, ff, circ_lo, circ_hi, bnew, flux);
    else if (lim == LIM_SUPERBEE) chain_whole<V, C, LIM_SUPERBEE>(vr, b, ff, circ_lo, circ_hi, bnew, flux);
    else chain_whole<V, C, LIM_MINMOD>(vr, b, ff, circ_lo, circ_hi, bnew, flux);
}

__device__ __forceinline__ float corner_velocity(float pm, float p, float rm, float r) { return (pm + p) * rcp_approx(rm + r); }
__device__ __forceinline__ double corner_velocity(double pm, double p, double rm, double r) { return quotient(pm + p, rm + r); }

// Chain kernel body.  Each thread reads its own C cells once (128-bit loads along x), forms their corner
// velocities and publishes them with B_I, 16 bytes a cell and lane, cell k of every thread in plane k
// (consecutive threads on consecutive 16 bytes, whichever way the sweep runs); after a barrier it reads
// the two cells on each side from its neighbours' planes, computes wMag of its own cells, publishes that
// too, and after a second barrier reads wMag of two cells on each side for the limited flux.  The window
// form without exchanges re-reads and re-divides all C + 8 cells of the chain's stencil from global memory in
// every thread (380 instructions a cell), which makes it instruction-bound.  64 registers a thread leave 32
// warps an SM; what bounds it now is the latency of its loads, along y and z also their 32-byte rows.
// Measured, chain and CT pass of one sweep on 256^3 cells in the mixed form: x 450 -> 205 us, y and z
// 552 -> 355 us; 512^2 (state in L2): y 20 -> 13 us.
template <typename T, int C>
__device__ __forceinline__ void mag_chain_win_body(const MagArgs& a, unsigned vblock) {
    extern __shared__ __align__(16) unsigned char smem[];
    using V = typename ChainLane<T>::V;
    using Rec = ChainRec<V>;
    constexpr int PASSES = ChainLane<T>::PASSES;
    const SweepGeom& g = a.sg;
    const int N = g.N, S = g.G, NT = g.CL > 1 ? g.NT : (int)blockDim.x, d = g.d;   // (blockDim: as in the fluid kernels)
    WinPos wp;
    wp.init(g, vblock);
    const int r0 = wp.s * C;
    const bool circ_lo = a.modeX[0] == BC_CIRC, circ_hi = a.modeX[1] == BC_CIRC;
    // local cells of the pencil's first and last rows (idle threads: no end near)
    const int lend = wp.colok ? -r0 : -64, hend = wp.colok ? N - 1 - r0 : 64;
    // own cells inside the pencil: fewer in a ragged last segment, none in idle threads
    const int nown = wp.colok ? (N - r0 < C ? N - r0 : C) : 0;
    // vector accesses along x need every segment to start on a multiple of C: pencils (and the arrays,
    // 256-byte aligned) start on one only where C divides N; ragged pencils go cell by cell
    const bool vec = d == 0 && N % C == 0;
    const int sd = (int)g.sd;
    const int o0 = wp.base + r0 * sd;
    pdl_wait();
    const DevTime* tm = a.tm;
    const int stop = tm->done | (g.CL == 1 ? tm->error : tm->halt);   // clusters: as in the fluid sweeps
    const T ff = (T)quotient_by(0.5 * tm->dt, a.dx, a.inv_dx);

    // ---- own cells: the corner velocity (magnetFlux.m:18-19) and B_I of both components ------------
    T vgo[2][C], bo[2][C];
    {
        T r[C], p[C], pm[2][C], rm[2][C];
        win_load<T, C>(a.w_rho, o0, sd, vec, nown, T(1), r);
        win_load<T, C>(a.w_pX, o0, sd, vec, nown, T(0), p);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int ie = a.first[q] ? wp.c1 : wp.c2;
            const int nbp = trans_offset(a, q, ie, -1, a.modeI_mom[q][0]);    // p_X: mom class
            const int nbr = trans_offset(a, q, ie, -1, a.modeI_mass[q][0]);   // rho: mass class
            win_load<T, C>(a.w_pX, o0 + nbp, sd, vec, nown, T(0), pm[q]);
            win_load<T, C>(a.w_rho, o0 + nbr, sd, vec, nown, T(1), rm[q]);
            win_load<T, C>(a.w_BI[q], o0, sd, vec, nown, T(0), bo[q]);
        }
        if (stop) return;   // after the loads are on their way: the flags take as long as they do
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int k = 0; k < C; ++k) vgo[q][k] = corner_velocity(pm[q][k], p[k], rm[q][k], r[k]);
    }
    V bn[PASSES][C], fl[PASSES][C];
    auto lane = [&](const T (&x)[2][C], int ps, int k) -> V {
        if constexpr (PASSES == 1) return F2(x[0][k], x[1][k]);
        else return x[ps][k];
    };
    if (S == 1 && N == C) {   // the whole pencil in this thread (uniform over the launch): nothing to exchange
#pragma unroll
        for (int ps = 0; ps < PASSES; ++ps) {
            V vr[C], b[C];
#pragma unroll
            for (int k = 0; k < C; ++k) { vr[k] = lane(vgo, ps, k); b[k] = lane(bo, ps, k); }
            chain_whole_lim<V, C>(a.limiter, vr, b, v_splat<V>((double)ff), circ_lo, circ_hi, bn[ps], fl[ps]);
        }
    } else {
        Rec* X = reinterpret_cast<Rec*>(smem);
        const int t = threadIdx.x;
#pragma unroll
        for (int ps = 0; ps < PASSES; ++ps)
#pragma unroll
            for (int k = 0; k < C; ++k) {
                Rec rc;
                rc.vg = lane(vgo, ps, k);
                rc.b = lane(bo, ps, k);
                X[(ps * C + k) * NT + t] = rc;
            }
        win_barrier(g);
        const int ls = d == 0 ? 1 : g.Wb;   // thread distance between consecutive segments of a pencil
        // the segments on both sides: in this CTA and whole (one wrap at most under circ ends), or found row by
        // row (const ends, a ragged last segment, another CTA of the cluster)
        const bool whole = N % C == 0;
        int nb[2];
        bool fast = true;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            int sm = wp.s + (m ? 1 : -1);
            if (g.CL == 1 && whole && circ_lo && circ_hi) sm = sm < 0 ? sm + S : (sm >= S ? sm - S : sm);
            nb[m] = t + (sm - wp.s) * ls;
            fast = fast && sm >= 0 && (sm < S - 1 || (whole && sm == S - 1));
            if (g.CL > 1) fast = fast && nb[m] >= 0 && nb[m] < NT;
        }
        fast = (fast && nown == C) || !wp.colok;   // idle threads: any address of the CTA will do
#pragma unroll
        for (int m = 0; m < 2; ++m) nb[m] = wp.colok ? nb[m] : t;
        const int rank = g.CL > 1 ? wp.s / NT : 0;
        // the record of window cell j in a set of planes, through its row
        auto find = [&](auto* P, int j, int ps) {
            const int r = win_row_multi(r0 + j, N, circ_lo, circ_hi);
            const int sg = r / C, k = r - sg * C;
            if (g.CL > 1) {
                const int rk = sg / NT;
                if (rk != rank) P = cg::this_cluster().map_shared_rank(P, rk);
                return P[(ps * C + k) * NT + (sg - rk * NT)];
            }
            return P[(ps * C + k) * NT + t + (sg - wp.s) * ls];
        };
        const V ffv = v_splat<V>((double)ff);
        V* XW = reinterpret_cast<V*>(X + PASSES * C * NT);
        V vf[PASSES][C + 1], Wm[PASSES][C + 4];
#pragma unroll
        for (int ps = 0; ps < PASSES; ++ps) {
            V vr[C + 4], b[C + 2], wo[C];
#pragma unroll
            for (int k = 0; k < C; ++k) { vr[k + 2] = lane(vgo, ps, k); b[k + 1] = lane(bo, ps, k); }
#pragma unroll
            for (int j = -2; j < C + 2; ++j) {
                if (j >= 0 && j < C && (fast || j < nown)) continue;
                const int k = j < 0 ? j + C : j - C;   // the fast path's plane
                const Rec rc = fast ? X[(ps * C + (k >= 0 && k < C ? k : 0)) * NT + nb[j < 0 ? 0 : 1]] : find(X, j, ps);
                vr[j + 2] = rc.vg;
                if (j >= -1 && j < C + 1) b[j + 1] = rc.b;
            }
            // only segments at a const end pay for its fills
            if ((!circ_lo && lend == 0) || (!circ_hi && hend < C))
                chain_predict<V, C, true>(vr, b, ffv, circ_lo, circ_hi, lend, hend, wo, vf[ps]);
            else
                chain_predict<V, C, false>(vr, b, ffv, circ_lo, circ_hi, lend, hend, wo, vf[ps]);
#pragma unroll
            for (int k = 0; k < C; ++k) {
                XW[(ps * C + k) * NT + t] = wo[k];
                Wm[ps][k + 2] = wo[k];
            }
        }
        win_barrier(g);
#pragma unroll
        for (int ps = 0; ps < PASSES; ++ps) {
            V b[C];
#pragma unroll
            for (int k = 0; k < C; ++k) b[k] = lane(bo, ps, k);
#pragma unroll
            for (int j = -2; j < C + 2; ++j) {
                if (j >= 0 && j < C && (fast || j < nown)) continue;
                const int k = j < 0 ? j + C : j - C;
                Wm[ps][j + 2] = fast ? XW[(ps * C + (k >= 0 && k < C ? k : 0)) * NT + nb[j < 0 ? 0 : 1]] : find(XW, j, ps);
            }
            chain_correct_lim<V, C>(a.limiter, Wm[ps], vf[ps], b, ffv, !circ_lo && lend == 0, bn[ps], fl[ps]);
        }
        if (g.CL > 1) cluster_sync();   // the other ranks have read this CTA's planes before it exits
    }
    pdl_trigger();
    // B_I in place (each thread's own rows, read by nobody else) and the limited flux for the CT pass
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        T bq[C], fq[C];
#pragma unroll
        for (int k = 0; k < C; ++k) {
            if constexpr (PASSES == 1) {
                float x[2], y[2];
                bn[0][k].get(x[0], x[1]);
                fl[0][k].get(y[0], y[1]);
                bq[k] = x[q];
                fq[k] = y[q];
            } else {
                bq[k] = bn[q][k];
                fq[k] = fl[q][k];
            }
        }
        if (wp.colok) {
            win_store<T, C>(a.w_BI[q], o0, sd, vec, nown, bq);
            win_store<T, C>(q ? a.F[1] : a.F[0], o0, sd, vec, nown, fq);
        }
    }
}

// CT pass body.  D_q at cell j is C_q at cell j - 1 and the cell-centred B_X at the last own cell needs the
// new B_X one cell further, so besides its own cells (128-bit loads along x) a thread reads C_q one row
// below and B_X one row above.
template <typename T, int C>
__device__ __forceinline__ void mag_ct_win_body(const MagArgs& a, unsigned vblock) {
    const SweepGeom& g = a.sg;
    const int N = g.N, d = g.d;
    WinPos wp;
    wp.init(g, vblock);
    const int r0 = wp.colok ? wp.s * C : 0;
    const bool circ_lo = a.modeX[0] == BC_CIRC, circ_hi = a.modeX[1] == BC_CIRC;
    const int nown = wp.colok ? (N - r0 < C ? N - r0 : C) : 0;
    const bool vec = d == 0 && N % C == 0;   // as in the chain
    const int sd = (int)g.sd;
    const int o0 = wp.base + r0 * sd;
    // the rows below and above the segment: wrapped, or the end row itself (const: C_q and B_X copy their
    // end values)
    const int olo = r0 > 0 ? o0 - sd : (circ_lo ? wp.base + (N - 1) * sd : o0);
    const bool past = r0 + nown >= N;
    const int ohi = past ? wp.base + (circ_hi ? 0 : (N - 1) * sd) : o0 + nown * sd;
    const bool end_hi = !circ_hi && past;
    pdl_wait();
    const DevTime* tm = a.tm;
    const int stop = tm->done | (g.CL == 1 ? tm->error : tm->halt);   // clusters: as in the fluid sweeps
    const double dt = tm->dt;
    T* BX = reinterpret_cast<T*>(a.w_BX);
    // C_q = F_q - F_q.shift(I_q, +1) (relaxingMagnet.m:56) at cells -1 .. C-1 (index j + 1)
    T f[2][C], fn[2][C], fl[2], fln[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const T* F = reinterpret_cast<const T*>(q ? a.F[1] : a.F[0]);
        const int nb = trans_offset(a, q, a.first[q] ? wp.c1 : wp.c2, +1, a.modeI_mag[q][1]);
        win_load<T, C>(F, o0, sd, vec, nown, T(0), f[q]);
        win_load<T, C>(F, o0 + nb, sd, vec, nown, T(0), fn[q]);
        fl[q] = F[olo];
        fln[q] = F[olo + nb];
    }
    T bxo[C];
    win_load<T, C>(BX, o0, sd, vec, nown, T(0), bxo);
    const T bxn = BX[ohi];
    // cell-centred B_I2 needs B_I2 at the pencil and its I2+1 neighbour (read only here)
    const int nb2 = trans_offset(a, 1, a.first[1] ? wp.c1 : wp.c2, +1, a.modeI_mag[1][1]);
    T b2[C], b2n[C];
    win_load<T, C>(a.w_BI[1], o0, sd, vec, nown, T(0), b2);
    win_load<T, C>(a.w_BI[1], o0 + nb2, sd, vec, nown, T(0), b2n);
    if (stop) return;
    T Cq[2][C + 1];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        Cq[q][0] = fl[q] - fln[q];
#pragma unroll
        for (int k = 0; k < C; ++k) Cq[q][k + 1] = f[q][k] - fn[q][k];
    }
    win_barrier(g);   // every thread has read B_X before any writes it
    // D_q = C_q.shift(X,-1); B_X = (B_X - dt/dI1 D_1) - dt/dI2 D_2 at the own cells and the one after them
    const T f0 = (T)quotient_by(dt, a.dI[0], a.inv_dI[0]), f1 = (T)quotient_by(dt, a.dI[1], a.inv_dI[1]);
    T bx[C], cbx[C], cb2[C];
#pragma unroll
    for (int k = 0; k < C; ++k) bx[k] = v_fma(-f1, Cq[1][k], v_fma(-f0, Cq[0][k], bxo[k]));
#pragma unroll
    for (int k = 0; k < C; ++k) {
        // the new B_X one cell up: the next own cell's, or past the last own cell the row above's (its D_q is
        // C_q of this cell); B_X.shift(X, +1) past a const end is the end cell's value
        T up = v_fma(-f1, Cq[1][k + 1], v_fma(-f0, Cq[0][k + 1], bxn));
        if (end_hi) up = bx[k];
        if (k + 1 < C && k + 1 < nown) up = bx[k + 1 < C ? k + 1 : k];
        cbx[k] = T(0.5) * (bx[k] + up);
        cb2[k] = T(0.5) * (b2[k] + b2n[k]);
    }
    pdl_trigger();
    if (!wp.colok) return;
    win_store<T, C>(BX, o0, sd, vec, nown, bx);
    win_store<T, C>(a.w_CBX, o0, sd, vec, nown, cbx);
    win_store<T, C>(a.w_CB2, o0, sd, vec, nown, cb2);
}

// The chain of up to 4 cells per thread in the mixed form fits 64 registers, so two 512-thread CTAs (32 warps)
// share an SM and cover one another's loads and barriers.
template <typename T, int C>
constexpr int chain_min_blocks() { return sizeof(T) == 4 && C <= 4 ? 2 : 1; }

template <typename T, int C>
__global__ void __launch_bounds__(512, chain_min_blocks<T, C>()) mag_chain_win_kernel(const __grid_constant__ MagArgs a) {
    mag_chain_win_body<T, C>(a, blockIdx.x);
}

template <typename T, int C>
__global__ void __launch_bounds__(512, chain_min_blocks<T, C>()) mag_ct_win_kernel(const __grid_constant__ MagArgs a) {
    mag_ct_win_body<T, C>(a, blockIdx.x);
}

template <typename T, int C>
__global__ void __launch_bounds__(512, chain_min_blocks<T, C>()) mag_chain_win_batch_kernel(const MagArgs* __restrict__ args,
                                                                      const BlockMap* __restrict__ map) {
    __shared__ MagArgs sa;
    const BlockMap bm = map[blockIdx.x];
    load_member_args(sa, args + bm.member);
    __syncthreads();
    mag_chain_win_body<T, C>(sa, (unsigned)bm.block);
}

template <typename T, int C>
__global__ void __launch_bounds__(512, chain_min_blocks<T, C>()) mag_ct_win_batch_kernel(const MagArgs* __restrict__ args,
                                                                   const BlockMap* __restrict__ map) {
    __shared__ MagArgs sa;
    const BlockMap bm = map[blockIdx.x];
    load_member_args(sa, args + bm.member);
    __syncthreads();
    mag_ct_win_body<T, C>(sa, (unsigned)bm.block);
}

}  // namespace img
