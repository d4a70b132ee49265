// fxb_march3d.cuh -- the sweeps of the 3-D step with the default options as
// one kernel per direction: slopes, face states and Riemann fluxes.  (The
// extended-option kernels and the persistent AMR kernel run the per-stage
// kernels of fxb_hydro3d.cuh.)
//
// What bounds them is latency, not HBM: an FP64 face state is a chain of some
// 2,000 instructions, and registers and shared memory leave three CTAs of 128
// threads per SM.  So the point of the shape is that nothing in the chain
// waits for memory: a thread of the y and z sweeps walks along its line, what
// the next cell needs of this one (the stencil's cells, two limited slopes,
// the right-face state) stays in the thread's own slots of shared memory, the
// line's next cell is loaded into registers and the cell's sigmas are copied
// into shared memory (cp.async) before the Riemann solve of the previous
// face, and there is no barrier in the loop.  Neighbouring threads own
// neighbouring x, so every access is coalesced.  The face states and slopes
// never go through HBM (PPM FP64: 2.7 instead of 3.9 GB per 128^3 step).
//
// Against slope, face-state and flux kernels (FP64) and the fused tile kernel
// with two barriers per cell (FP32), 128^3: one direction of PPM FP64 374 ->
// 249 us along y and z and 398 -> 324 us along x, of WENO5 FP64 470 -> 407 to 419
// and 467 us, PPM FP32 190 -> 123 and 162 us; without the copies ahead the y and z
// kernels took 390 us.  Whole steps, with the rest of the step as it is now
// (sweeps side by side, boundary fluxes from here): PPM 1.36 -> 1.04 ms (mixed
// 0.77 -> 0.56), WENO5 with gravity 1.58 -> 1.49 (mixed 0.82 -> 0.61), AMR (288
// leaves of 16^3) 0.99 -> 0.82 (mixed 0.55 -> 0.43).
#pragma once
#include "fxb_hydro3d.cuh"
#include "fxb_tma.cuh"

#include <type_traits>

namespace fxb {

template <class S> __device__ __forceinline__ void cp_async(S *dst, const S *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"((int)sizeof(S))
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// The sigmas a face state of direction DIR reads, as six groups of six values:
// those of the two transverse directions SA and SB at the cell, and for the
// CTU terms sigma_SA one cell before and behind along EA, sigma_SB along EB.
template <int DIR> struct SweepSig {
    static constexpr int EA = (DIR + 1) % 3, SA = (DIR + 2) % 3, EB = (DIR + 2) % 3, SB = (DIR + 1) % 3;
};
// address of group g of the cell with padded index (i, j, k)
template <int DIR, class R>
__device__ __forceinline__ const R *sweep_sig_at(const R *sig, const Grid3 &G, int g, int i, int j, int k)
{
    using Q = SweepSig<DIR>;
    int di = 0, dj = 0, dk = 0;
    if (g >= 2) offs(g < 4 ? Q::EA : Q::EB, g & 1 ? 1 : -1, di, dj, dk);
    return sig + tile_at<NSIG>(G.pidx(i + di, j + dj, k + dk)) + 6 * TILE3 * (g == 0 || g == 2 || g == 3 ? Q::SA : Q::SB);
}

// The face states of one cell from its interface values: flattening,
// characteristic tracing, transverse terms, negativity fallback, gravity and
// the full-CTU terms, as face_states_tail and face_states_finish.  C: the
// cell's sweep-order primitives; q: dt / del along the sweep, dt / 2 del of the
// three axes, the CTU factor; sg(g, v): value v of sigma group g (SweepSig);
// ready(): called once before the first sg.
template <class R, bool AMR, int DIR, int OPT, class SG, class READY>
__device__ __forceinline__ void sweep_states(const Args3D &a, const Ctx3<R, AMR> &X, const double q[5], double dt, int i,
                                             int j, int k, const R C[6], const EigBase<R> &eb, const Eig<R> &e,
                                             R vecL[6], R vecR[6], SG sg, READY ready, R Wm[6], R Wp[6])
{
    using Q = SweepSig<DIR>;
    const Grid3 &G = X.G;
    if (a.prm.flattening) flatten(X.flat[(long)DIR * G.npad() + G.pidx(i, j, k)], C, vecL, vecR);
    R wm[6], wp[6], g[6];
    ppm_trace(e, R(q[0]), R(0.5 * q[0]), C, vecL, vecR, wm, wp);
    unrot3(DIR, wm, Wm); unrot3(DIR, wp, Wp); unrot3(DIR, C, g);
    ready();
    // transverse terms of the lower axis first (hy_dataReconstOneStep.F90:931-962)
    constexpr bool a_first = Q::SA < Q::SB;
    const R h1 = R(q[1 + (a_first ? Q::SA : Q::SB)]), h2 = R(q[1 + (a_first ? Q::SB : Q::SA)]);
#pragma unroll
    for (int v = 0; v < 6; v++) {
        const R s1 = h1 * sg(a_first ? 0 : 1, v), s2 = h2 * sg(a_first ? 1 : 0, v);
        Wm[v] = Wm[v] - s1; Wp[v] = Wp[v] - s1;
        Wm[v] = Wm[v] - s2; Wp[v] = Wp[v] - s2;
    }
    const bool bad = Wm[0] < R(0) || Wp[0] < R(0) || Wm[4] < R(0) || Wp[4] < R(0);
#pragma unroll
    for (int v = 0; v < 6; v++) { Wm[v] = bad ? g[v] : Wm[v]; Wp[v] = bad ? g[v] : Wp[v]; }
    if (a.prm.use_gravity) {   // hy_getRiemannState.F90:843-885
        const R hdt = R(0.5 * dt);
        R gl, gr;
        gravity_face_values(a.prm, DIR, gl, gr);
#pragma unroll
        for (int v = 0; v < 3; v++) {
            Wp[1 + v] = Wp[1 + v] + hdt * (v == DIR ? gr : R(a.prm.grav[v]));
            Wm[1 + v] = Wm[1 + v] + hdt * (v == DIR ? gl : R(a.prm.grav[v]));
        }
    }
    if (a.prm.use_3d_full_ctu) {
        const bool aux = OPT == OPT_DEFAULT || a.prm.use_aux_eint != 0;
        R T[6], U[6], m[6], c[6], p[6], r[6];
        auto term = [&](int ax, int g0, int gm, int gp, R out[6]) {
            R sm[6], sc[6], sp[6];
#pragma unroll
            for (int v = 0; v < 6; v++) { sm[v] = sg(gm, v); sc[v] = sg(g0, v); sp[v] = sg(gp, v); }
            rot3(ax, sm, m); rot3(ax, sc, c); rot3(ax, sp, p);
            Eig<R> ev;
            eigen_dir(eb, g[1 + ax], ev);
            trans_flux(ev, m, c, p, aux, r);
            unrot3(ax, r, out);
        };
        term(Q::EA, 0, 2, 3, T);
        term(Q::EB, 1, 4, 5, U);
        const R f = R(q[4]);
#pragma unroll
        for (int v = 0; v < 6; v++) {
            Wp[v] = Wp[v] + (T[v] + U[v]) * f;
            Wm[v] = Wm[v] + (T[v] + U[v]) * f;
        }
        const bool low = Wp[0] <= R(0) || Wm[0] <= R(0) || Wp[4] <= R(0) || Wm[4] <= R(0);
#pragma unroll
        for (int v = 0; v < 6; v++) { Wm[v] = low ? g[v] : Wm[v]; Wp[v] = low ? g[v] : Wp[v]; }
    }
}

// the fluxes of a face of direction DIR into the flux array; on an AMR leaf
// also into its boundary fluxes (Grid_putFluxData) when the face is on the
// block's boundary (c = 0 or N; t1, t2: the face's transverse cell).  The
// pressure slot only where the update reads it (fp).
template <class R, bool AMR, int DIR>
__device__ __forceinline__ void store_fluxes(const Args3D &a, const Ctx3<R, AMR> &X, int i, int j, int k, bool fp,
                                             const R F[NF])
{
    R *f = X.flx[DIR] + tile_at<NF>(X.G.fidx(DIR, i, j, k));
#pragma unroll
    for (int q = 0; q < NF; q++) if (q != FP || fp) f[q * TILE3] = F[q];
    if constexpr (AMR) {
        const int c = DIR == 0 ? i : DIR == 1 ? j : k, N = DIR == 0 ? a.nx : DIR == 1 ? a.ny : a.nz;
        if (c == 0 || c == N) {
            const int t1 = DIR == 0 ? j : i, t2 = DIR == 2 ? j : k, n1 = DIR == 0 ? a.ny : a.nx;
            R *b = (R *)a.bflux + ((long)X.m.leaf * 6 + 2 * DIR + (c == N)) * NF * a.nfc + t2 * n1 + t1;
#pragma unroll
            for (int q = 0; q < NF; q++) if (q != FP || fp) b[q * a.nfc] = F[q];
        }
    }
}

// CTAs of T threads: 128, or on AMR leaves 64 where fewer threads are then
// without a line (8^3 leaves have 64 lines, 12^3 ones 144).  Resident CTAs per
// SM for 128 threads each: 168 registers per thread in FP64 (shared memory
// allows no fourth CTA), 96 in FP32 (six CTAs of 80 registers: PPM 128^3 0.66
// instead of 0.64 ms)
#ifndef FXB_MARCH_MINB64
#define FXB_MARCH_MINB64 3
#endif
#ifndef FXB_MARCH_MINB32
#define FXB_MARCH_MINB32 5
#endif
template <class R, int T> constexpr int march_resident()
{ return (sizeof(R) == 8 ? FXB_MARCH_MINB64 : FXB_MARCH_MINB32) * 128 / T; }
// per-thread slots: the stencil's cells (PPM 3, WENO5 5, six values each), two
// slopes (PPM), the previous cell's right-face state
template <int ORDER> struct MarchSlots {
    static constexpr int cells = ORDER == 5 ? 5 : 3;
    static constexpr int slope = cells * 6, wp = slope + (ORDER == 5 ? 0 : 12), sig = wp + 6, value = sig + 36;
};

template <class R, int ORDER, bool AMR, int DIR, int OPT, int T>
__global__ void __launch_bounds__(T, march_resident<R, T>()) march3d_kernel(const Args3D a)
{
    static_assert(DIR == 1 || DIR == 2, "lines along y or z");
    extern __shared__ __align__(16) unsigned char march_smem[];
    __shared__ double sq[6];
    R *const sl = reinterpret_cast<R *>(march_smem) + threadIdx.x;
    const Ctx3<R, AMR> X(a, blockIdx.z);
    const Grid3 &G = X.G;
    const double dt = a.dtv ? a.dtv[0] : a.dt_arg;
    // the step's quotients: dt / del along the line, dt / 2 del per axis, dt^2 / 6 del del
    if (threadIdx.x < 5) {
        const double del = DIR == 1 ? X.dy : X.dz;
        sq[threadIdx.x] = threadIdx.x == 0 ? dt / del
                          : threadIdx.x == 1 ? 0.5 * dt / X.dx
                          : threadIdx.x == 2 ? 0.5 * dt / X.dy
                          : threadIdx.x == 3 ? 0.5 * dt / X.dz
                                             : dt * dt / (DIR == 1 ? 6. * X.dz * X.dx : 6. * X.dx * X.dy);
    }
    __syncthreads();
    const bool fp = a.prm.fpres != 1.0;            // else the update does not read the pressure slot
    const int N = DIR == 1 ? a.ny : a.nz, N2 = DIR == 1 ? a.nz : a.ny;
    const int line = (int)(blockIdx.x * T + threadIdx.x);
    if (line >= a.nx * N2) return;
    const int t2 = (int)fast_div((unsigned)line, a.fdx[0]), i = line - t2 * a.nx;
    const int f0 = (int)blockIdx.y * a.march_len, f1 = min(f0 + a.march_len, N + 1);

    // the line's cells in the source arrays
    const int stride = DIR == 1 ? X.sx : X.sx * X.sy;
    const R *srcR = X.srcR;
    const double *src = X.src;
    const long base = AMR ? (DIR == 1 ? (long)(t2 + X.so) * X.sy * X.sx + X.so * X.sx
                                      : (long)X.so * X.sy * X.sx + (long)(t2 + X.so) * X.sx) + i + X.so
                          : (DIR == 1 ? (long)t2 * X.sy * X.sx : (long)t2 * X.sx) + i;
    if constexpr (AMR) srcR += base; else src += base;
    constexpr int v1 = VX + DIR, v2 = VX + (DIR + 1) % 3, v3 = VX + (DIR + 2) % 3;
    // sweep-order primitives (D, v1, v2, v3, P, EI) and gamc of cell c
    auto load = [&](int c, R v[6], R &gc) {
        if constexpr (AMR) {
            const R *p = srcR + (long)c * stride;
            v[0] = __ldg(p + D * X.svs); v[1] = __ldg(p + v1 * X.svs); v[2] = __ldg(p + v2 * X.svs);
            v[3] = __ldg(p + v3 * X.svs); v[4] = __ldg(p + P * X.svs); v[5] = __ldg(p + EI * X.svs);
            gc = __ldg(p + GC * X.svs);
        } else {
            double s = 1.0;
            const int m = map_axis(c, N, a.bc[2 * DIR], a.bc[2 * DIR + 1], &s);
            const double *p = src + (long)m * stride;
            v[0] = (R)__ldg(p + D * X.svs); v[1] = (R)(__ldg(p + v1 * X.svs) * s); v[2] = (R)__ldg(p + v2 * X.svs);
            v[3] = (R)__ldg(p + v3 * X.svs); v[4] = (R)__ldg(p + P * X.svs); v[5] = (R)__ldg(p + EI * X.svs);
            gc = (R)__ldg(p + GC * X.svs);
        }
    };
    // the two Eos gammas of cell c, for the Riemann solver
    auto load_gammas = [&](int c, R &gc, R &ge) {
        if constexpr (AMR) {
            const R *p = srcR + (long)c * stride;
            gc = __ldg(p + GC * X.svs); ge = __ldg(p + GE * X.svs);
        } else {
            double s = 1.0;
            const double *p = src + (long)map_axis(c, N, a.bc[2 * DIR], a.bc[2 * DIR + 1], &s) * stride;
            gc = (R)__ldg(p + GC * X.svs); ge = (R)__ldg(p + GE * X.svs);
        }
    };
    using SL = MarchSlots<ORDER>;
    auto put = [&](int slot, const R v[6]) {
#pragma unroll
        for (int q = 0; q < 6; q++) sl[(slot + q) * T] = v[q];
    };
    auto get = [&](int slot, R v[6]) {
#pragma unroll
        for (int q = 0; q < 6; q++) v[q] = sl[(slot + q) * T];
    };

    // ring of the stencil's cells: ring[0] is the oldest
    int ring[SL::cells];
#pragma unroll
    for (int q = 0; q < SL::cells; q++) ring[q] = 6 * q;
    int dbm = SL::slope, dbc = SL::slope + 6;      // slopes of the cell before and of the cell
    EigBase<R> eb;                                 // PPM: of the cell, from the slope of the iteration before
    R gcp = R(0);                                  // PPM: gamc of the cell behind
    const int c0 = f0 - 1;
    {
        R A[6], B[6], C[6], g;
        if constexpr (ORDER == 3) {
            R Dn[6], gb, gcc, db[6];
            load(c0 - 2, A, g); load(c0 - 1, B, gb); load(c0, C, gcc); load(c0 + 1, Dn, gcp);
            Eig<R> e;
            if (!eigen(B[0], B[1], B[4], gb, e)) atomicOr(a.err, ERR_SOUND);
            tvd_slope<R, OPT>(a.prm, e, A, B, C, db);
            put(dbm, db);
            if (!eigen_base(C[0], C[4], gcc, eb)) atomicOr(a.err, ERR_SOUND);
            eigen_dir(eb, C[1], e);
            tvd_slope<R, OPT>(a.prm, e, B, C, Dn, db);
            put(dbc, db);
            put(ring[0], B); put(ring[1], C); put(ring[2], Dn);
        } else {
            // cells c0 - 2 .. c0 + 1; the iteration loads the fifth
#pragma unroll
            for (int o = 0; o < 4; o++) { load(c0 - 2 + o, A, g); put(ring[o], A); }
        }
    }
    R Wm[6], Wp[6], gcl = R(0), gel = R(0), gc = R(0), ge = R(0);
    for (int c = c0;; c++) {
        // loads of the next cell and of this cell's gammas, ahead of the
        // Riemann solve of the previous face
        R E[6], gE = R(0), gcn = R(0), gen = R(0);
        if (c < f1) {
            load(c + 2, E, gE);
            load_gammas(c, gcn, gen);
            const int j = DIR == 1 ? c : t2, k = DIR == 2 ? c : t2;
#pragma unroll
            for (int g = 0; g < 6; g++) {
                if (g >= 2 && !a.prm.use_3d_full_ctu) continue;
                const R *p = sweep_sig_at<DIR>((const R *)X.sig, G, g, i, j, k);
#pragma unroll
                for (int v = 0; v < 6; v++) cp_async(sl + (SL::sig + 6 * g + v) * T, p + v * TILE3);
            }
            cp_async_commit();
        }
        if (c > f0) {
            // face c - 1: Wp of cell c - 2 against Wm of cell c - 1
            R VL[6], F[NF];
            get(SL::wp, VL);
            const int er = riemann<R, 0, OPT>(a.prm, DIR, VL, gcl, gel, Wm, gc, ge, F);
            if (er) atomicOr(a.err, er);
            store_fluxes<R, AMR, DIR>(a, X, i, DIR == 1 ? c - 1 : t2, DIR == 1 ? t2 : c - 1, fp, F);
        }
        if (c == f1) break;
        if (c > c0) put(SL::wp, Wp);               // of cell c - 1
        gcl = gc; gel = ge;
        gc = gcn; ge = gen;
        const int j = DIR == 1 ? c : t2, k = DIR == 2 ? c : t2;
        R vecL[6], vecR[6], Vc[6];
        EigBase<R> ebc;
        Eig<R> e;
        if constexpr (ORDER == 3) {
            R Vm[6], Vp[6], dbN[6], db0[6], dbP[6];
            get(ring[1], Vc); get(ring[2], Vp);
            ebc = eb;
            if (!eigen_base(Vp[0], Vp[4], gcp, eb)) atomicOr(a.err, ERR_SOUND);
            eigen_dir(eb, Vp[1], e);
            tvd_slope<R, OPT>(a.prm, e, Vc, Vp, E, dbP);
            gcp = gE;
            get(ring[0], Vm);
            get(dbm, dbN); get(dbc, db0);
            ppm_interfaces(Vm, Vc, Vp, dbN, db0, dbP, vecL, vecR);
            put(dbm, dbP);
            const int t = dbm; dbm = dbc; dbc = t;
            put(ring[0], E);
            const int r0 = ring[0]; ring[0] = ring[1]; ring[1] = ring[2]; ring[2] = r0;
            eigen_dir(ebc, Vc[1], e);
        } else {
            put(ring[4], E);
            get(ring[2], Vc);
            if (!eigen_base(Vc[0], Vc[4], gc, ebc)) atomicOr(a.err, ERR_SOUND);
            eigen_dir(ebc, Vc[1], e);
            weno_interfaces_of<R, OPT>(a.prm, e, [&](int v, int o) { return sl[(ring[o] + v) * T]; }, vecL, vecR);
            const int r0 = ring[0];
            ring[0] = ring[1]; ring[1] = ring[2]; ring[2] = ring[3]; ring[3] = ring[4]; ring[4] = r0;
        }
        sweep_states<R, AMR, DIR, OPT>(a, X, sq, dt, i, j, k, Vc, ebc, e, vecL, vecR,
                                       [&](int g, int v) { return sl[(SL::sig + 6 * g + v) * T]; },
                                       [] { cp_async_wait(); }, Wm, Wp);
        if (c >= f0 && c < N) {
            R *w = X.wst[DIR] + G.widx(DIR, i, j, k);
            const long nw = G.nw(DIR);
            w[0] = Wp[P];
            w[nw] = Wm[P];
        }
    }
}

// The number of pieces a line of `len` steps is cut into: each piece costs its
// own steps and `extra` more (a segment computes one cell's face states and two
// slopes more than it has faces), `units` CTAs work on each piece, `resident`
// run at a time, and up to eight waves of CTAs the last one counts whole.
inline int cut_line(int len, int least, double extra, long units, long resident)
{
    int best = 1;
    double cost = 1e300;
    const int most = len / least < 1 ? 1 : len / least;
    for (int n = 1; n <= most; n++) {
        const int piece = (len + n - 1) / n, pieces = (len + piece - 1) / piece;
        const double w = (double)units * pieces / resident;
        const double c = (w < 8. ? (double)(long)(w + 0.999999) : w + 0.5) * (piece + extra);
        if (c < 0.999 * cost) { cost = c; best = n; }
    }
    return best;
}
#ifndef FXB_MARCH_SMIN
#define FXB_MARCH_SMIN 3
#endif
// how one sweep is launched
struct SweepPlan {
    dim3 grid;
    int threads;
    size_t smem;
    double waves;              // its CTAs over those the chip holds at a time
};
template <class R, int ORDER, int DIR, int T> SweepPlan plan_march3d(Args3D &a, unsigned entries)
{
    const int N = DIR == 1 ? a.ny : a.nz, N2 = DIR == 1 ? a.nz : a.ny;
    const long ctas = ((long)a.nx * N2 + T - 1) / T, resident = 148L * march_resident<R, T>();
    long nseg = cut_line(N + 1, FXB_MARCH_SMIN, 1.5, ctas * entries, resident);
    a.march_len = (int)((N + nseg) / nseg);
    nseg = (N + a.march_len) / a.march_len;
    return {dim3((unsigned)ctas, (unsigned)nseg, entries), T, MarchSlots<ORDER>::value * T * sizeof(R),
            (double)ctas * nseg * entries / resident};
}

// ---- x sweep -------------------------------------------------------------------
// A CTA takes a tile of T1 lines along x, faces f0 .. f0 + Lx - 1 of each,
// and walks through planes of constant z.  Lanes run along x, so a line's
// neighbours are other threads: the window of the plane (T1 x (Lx + 5) cells
// of eight variables, three cells before the first face and two behind the
// last), the limited slopes and the right-face states pass through shared
// memory, with a barrier after each.  The window of the next plane is copied
// into the second buffer (cp.async) while this one is worked on.
#ifndef FXB_SWX_PMIN
#define FXB_SWX_PMIN 2
#endif
#ifndef FXB_SWX_MINB64
#define FXB_SWX_MINB64 3
#endif
#ifndef FXB_SWX_MINB32
#define FXB_SWX_MINB32 5
#endif
// CTAs of T threads: 160, or on AMR leaves 96 where a leaf's tiles then take
// fewer threads (8^3: one tile of 96); resident CTAs per SM
template <class R, int T> constexpr int swx_resident() { return (sizeof(R) == 8 ? FXB_SWX_MINB64 : FXB_SWX_MINB32) * 160 / T; }
// cells per line and tile beyond its faces: one more face state, and with PPM two more slopes
template <int ORDER> constexpr int swx_extra() { return ORDER == 3 ? 3 : 1; }
// FP64 copies the sigmas of the next plane into shared memory while it works
// on this one (RT 128^3 1.55 -> 1.51 ms per step, AMR 16^3 blocks 2.08 -> 2.01,
// before the sweeps ran side by side); FP32, with five CTAs per SM to switch
// between, reads them when it needs them (RT 128^3 0.69 ms then, 0.71 with the copies)
template <class R> constexpr bool swx_ahead() { return sizeof(R) == 8; }

template <class R, int ORDER, bool AMR, int OPT, int T>
__global__ void __launch_bounds__(T, swx_resident<R, T>()) sweepx3d_kernel(const Args3D a)
{
    using S = typename std::conditional<AMR, R, double>::type;    // type of the source arrays
    constexpr int EX = swx_extra<ORDER>();
    constexpr bool AHEAD = swx_ahead<R>();
    extern __shared__ __align__(16) unsigned char swx_smem[];
    __shared__ double sq[5];
    const Ctx3<R, AMR> X(a, blockIdx.z);
    const Grid3 &G = X.G;
    const int t = threadIdx.x;
    const double dt = a.dtv ? a.dtv[0] : a.dt_arg;
    const int T1 = a.swx_lines, Lx = a.swx_len, W = Lx + 5, NWIN = T1 * W, Lt = Lx + EX;
    S *const sV = reinterpret_cast<S *>(swx_smem);                // [2][8][T1][W]
    R *const sD = reinterpret_cast<R *>(sV + 16 * NWIN);          // PPM: [6][T] slopes
    R *const sW = sD + (ORDER == 3 ? 6 * T : 0);              // [6][T] right-face states
    // this thread's sigmas: sigma_y of the planes k - 1, k, k + 1 (six values
    // each, in turn), then sigma_z of plane k
    R *const sS = sW + 6 * T + threadIdx.x;
    // sigma_z of plane k of the lines before the tile's first and behind its
    // last one, [6][two lines of Lt cells in rows of T]
    R *const sH = sW + 30 * T;
    if (t < 5)
        sq[t] = t == 0 ? dt / X.dx
                : t == 1 ? 0.5 * dt / X.dx
                : t == 2 ? 0.5 * dt / X.dy
                : t == 3 ? 0.5 * dt / X.dz
                         : dt * dt / (6. * X.dy * X.dz);
    const bool fp = a.prm.fpres != 1.0;            // else the update does not read the pressure slot
    const int N = a.nx, N1 = a.ny, nseg = a.swx_segs;
    const int seg = blockIdx.x % nseg, f0 = seg * Lx, j0 = (blockIdx.x / nseg) * T1;
    const int k0 = blockIdx.y * a.swx_planes, k1 = min(k0 + a.swx_planes, a.nz);
    // copies of one plane's window: thread t takes window cells t and t + T
    // (cells behind the line's last one or beyond the last line repeat them)
    const S *src;
    if constexpr (AMR) src = X.srcR; else src = X.src;
    long woff[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int w = min(t + q * T, NWIN - 1), l = w / W;
        int x = min(f0 - 3 + w - l * W, N + 2);
        const int y = min(j0 + l, N1 - 1);
        double s_ = 1.0;
        if constexpr (!AMR) x = map_axis(x, N, a.bc[0], a.bc[1], &s_);
        woff[q] = (long)(y + X.so) * X.sx + x + X.so;
    }
    auto copy_plane = [&](int k, int buf) {
        const long z = (long)(k + X.so) * X.sy * X.sx;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int w = t + q * T;
            if (w < NWIN) {
#pragma unroll
                for (int v = 0; v < 8; v++) cp_async(sV + (buf * 8 + v) * NWIN + w, src + (v * X.svs + z + woff[q]));
            }
        }
        cp_async_commit();
    };
    const int l1 = t / Lt, ld = t - l1 * Lt;
    const int c = f0 - (ORDER == 3 ? 2 : 1) + ld, j = j0 + l1;    // this thread's cell and line
    const bool line = l1 < T1 && j < N1;
    const bool st = line && c >= f0 - 1 && c < f0 + Lx && c <= N;   // a face-state cell
    const int wc = l1 * W + c - (f0 - 3);                         // its place in the window
    // reflecting boundaries flip the normal velocity of the cells beyond them
    auto one_at = [&](const S *V, int v, int o) {
        const R x = (R)V[(v == 5 ? (int)EI : v) * NWIN + wc + o];
        if constexpr (AMR) return x;
        else return v == VX && (c + o < 0 ? a.bc[0] == 2 : c + o >= N && a.bc[1] == 2) ? x * R(-1) : x;
    };
    auto six_at = [&](const S *V, int o, R v[6]) {
#pragma unroll
        for (int q = 0; q < 6; q++) v[q] = one_at(V, q, o);
    };
    auto copy_sig = [&](int slot, int d, int k) {
        const R *p = (const R *)X.sig + tile_at<NSIG>(G.pidx(c, j, k)) + 6 * d * TILE3;
#pragma unroll
        for (int v = 0; v < 6; v++) cp_async(sS + (slot + v) * T, p + v * TILE3);
    };
    int rm = 0, rc = 6, rp = 12;       // slots of sigma_y of the planes k - 1, k, k + 1
    // sigma_z beside this line: the neighbour thread's own, or the outer lines'
    const bool first = l1 == 0, last = l1 + 1 == T1 || j + 1 == N1;
    const R *const hm = first ? sH + ld : sS - Lt + 18 * T, *const hp = last ? sH + Lt + ld : sS + Lt + 18 * T;
    auto copy_sigz = [&](int k) {
        copy_sig(18, 2, k);
#pragma unroll
        for (int side = 0; side < 2; side++) {
            if (side ? !last : !first) continue;
            const R *p = sweep_sig_at<0>((const R *)X.sig, G, 2 + side, c, j, k);
#pragma unroll
            for (int v = 0; v < 6; v++) cp_async(sH + v * T + side * Lt + ld, p + v * TILE3);
        }
    };
    copy_plane(k0, 0);
    if (AHEAD && st) {
        copy_sig(rm, 1, k0 - 1); copy_sig(rc, 1, k0); copy_sig(rp, 1, k0 + 1);
        copy_sigz(k0);
        cp_async_commit();
    }
    for (int k = k0; k < k1; k++) {
        const int buf = (k - k0) & 1;
        cp_async_wait();
        __syncthreads();               // the window of this plane is there, the other buffer is free
        if (k + 1 < k1) copy_plane(k + 1, buf ^ 1);
        const S *V = sV + buf * 8 * NWIN;
        R Wm[6], Wp[6], Vc[6], vecL[6], vecR[6];
        EigBase<R> eb;
        Eig<R> e;
        if constexpr (ORDER == 3) {
            if (line && c <= N + 1) {
                R Vm[6], Vp[6], db[6];
                six_at(V, -1, Vm); six_at(V, 0, Vc); six_at(V, 1, Vp);
                if (!eigen_base(Vc[0], Vc[4], (R)V[GC * NWIN + wc], eb)) atomicOr(a.err, ERR_SOUND);
                eigen_dir(eb, Vc[1], e);
                tvd_slope<R, OPT>(a.prm, e, Vm, Vc, Vp, db);
#pragma unroll
                for (int q = 0; q < 6; q++) sD[q * T + t] = db[q];
            }
            __syncthreads();
            if (st) {
                R Vm[6], Vp[6], dbN[6], db0[6], dbP[6];
                six_at(V, -1, Vm); six_at(V, 1, Vp);
#pragma unroll
                for (int q = 0; q < 6; q++) {
                    dbN[q] = sD[q * T + t - 1]; db0[q] = sD[q * T + t]; dbP[q] = sD[q * T + t + 1];
                }
                ppm_interfaces(Vm, Vc, Vp, dbN, db0, dbP, vecL, vecR);
            }
        } else if (st) {
            six_at(V, 0, Vc);
            if (!eigen_base(Vc[0], Vc[4], (R)V[GC * NWIN + wc], eb)) atomicOr(a.err, ERR_SOUND);
            eigen_dir(eb, Vc[1], e);
            weno_interfaces_of<R, OPT>(a.prm, e, [&](int v, int o) { return one_at(V, v, o - 2); }, vecL, vecR);
        }
        if (st) {
            const R *gp[6];
            R own[12];
#pragma unroll
            for (int g = 0; g < 6; g++) gp[g] = sweep_sig_at<0>((const R *)X.sig, G, g, c, j, k);
            if (!AHEAD) {
#pragma unroll
                for (int v = 0; v < 12; v++) own[v] = __ldg(gp[v / 6] + v % 6 * TILE3);
            }
            const int at[6] = {18, rc, 0, 0, rm, rp};
            auto sg = [&](int g, int v) {
                if (AHEAD) return g == 2 ? hm[v * T] : g == 3 ? hp[v * T] : sS[(at[g] + v) * T];
                return g < 2 ? own[6 * g + v] : __ldg(gp[g] + v * TILE3);
            };
            sweep_states<R, AMR, 0, OPT>(a, X, sq, dt, c, j, k, Vc, eb, e, vecL, vecR, sg, [] {}, Wm, Wp);
#pragma unroll
            for (int q = 0; q < 6; q++) sW[q * T + t] = Wp[q];
            if (c >= f0 && c < N) {
                R *w = X.wst[0] + G.widx(0, c, j, k);
                w[0] = Wp[P];
                w[G.nw(0)] = Wm[P];
            }
        }
        __syncthreads();
        if (AHEAD && st && k + 1 < k1) {   // the next plane's sigmas, over the ones just used
            copy_sig(rm, 1, k + 2);
            copy_sigz(k + 1);
            cp_async_commit();
        }
        {
            const int r = rm; rm = rc; rc = rp; rp = r;
        }
        if (st && c >= f0) {
            R VL[6], F[NF];
#pragma unroll
            for (int q = 0; q < 6; q++) VL[q] = sW[q * T + t - 1];
            const int er = riemann<R, 0, OPT>(a.prm, 0, VL, (R)V[GC * NWIN + wc - 1], (R)V[GE * NWIN + wc - 1], Wm,
                                         (R)V[GC * NWIN + wc], (R)V[GE * NWIN + wc], F);
            if (er) atomicOr(a.err, er);
            store_fluxes<R, AMR, 0>(a, X, c, j, k, fp, F);
        }
    }
}

// The tile of a CTA of T threads: of up to 16 lines (no more than there are)
// the count with the fewest tiles per plane, the line's faces split evenly
// over the segments.
template <class R, int ORDER, bool AMR, int T> SweepPlan plan_sweepx3d(Args3D &a, unsigned entries)
{
    constexpr int EX = swx_extra<ORDER>();
    long tiles = -1;
    // (two lines at least where the tile's outer lines share rows of T values)
    for (int t1 = swx_ahead<R>() ? 2 : 1; t1 <= 16 && (t1 <= 2 || t1 <= a.ny); t1++) {
        int len = T / t1 - EX;
        len = len < a.nx + 1 ? len : a.nx + 1;
        if (len < 2 || t1 * (len + 5) > 2 * T) continue;
        const int segs = (a.nx + len) / len;
        const long n = (long)segs * ((a.ny + t1 - 1) / t1);
        if (tiles < 0 || n <= tiles) {
            tiles = n;
            a.swx_lines = t1;
            a.swx_segs = segs;
            a.swx_len = (a.nx + segs) / segs;
        }
    }
    const long resident = 148L * swx_resident<R, T>();
    long chunks = cut_line(a.nz, FXB_SWX_PMIN, 1., tiles * entries, resident);
    a.swx_planes = (int)((a.nz + chunks - 1) / chunks);
    chunks = (a.nz + a.swx_planes - 1) / a.swx_planes;
    const size_t smem = 16 * (size_t)a.swx_lines * (a.swx_len + 5) * (AMR ? sizeof(R) : sizeof(double)) +
                        ((ORDER == 3 ? 12 : 6) + (swx_ahead<R>() ? 30 : 0)) * (size_t)T * sizeof(R);
    return {dim3((unsigned)tiles, (unsigned)chunks, entries), T, smem, (double)tiles * chunks * entries / resident};
}

// the plan of the sweep of direction DIR; its numbers into a
template <class R, int ORDER, bool AMR, int DIR> SweepPlan plan_sweep3d(Args3D &a, unsigned entries)
{
    if constexpr (AMR) {
        // the CTA size that leaves fewer threads of a leaf idle: us per step,
        // 160 and 128 threads / the choice, 1,184 leaves of 8^3 PPM 654 / 623
        // (FP32 340 / 317), WENO5 914 / 788 (374 / 338), 288 of 12^3 PPM 516 / 445
        // (270 / 247).  FP32 keeps the larger where one piece of every
        // line fills a quarter of the chip at most (64 leaves of 8^3: van Leer
        // 45, 48 with the smaller).
        Args3D b = a;
        SweepPlan wide, narrow;
        if constexpr (DIR == 0) {
            wide = plan_sweepx3d<R, ORDER, AMR, 160>(a, entries);
            narrow = plan_sweepx3d<R, ORDER, AMR, 96>(b, entries);
        } else {
            wide = plan_march3d<R, ORDER, DIR, 128>(a, entries);
            narrow = plan_march3d<R, ORDER, DIR, 64>(b, entries);
        }
        if ((sizeof(R) == 4 && wide.waves <= 0.25 * wide.grid.y) ||
            (long)narrow.threads * narrow.grid.x >= (long)wide.threads * wide.grid.x) return wide;
        a = b;
        return narrow;
    } else if constexpr (DIR == 0) {
        return plan_sweepx3d<R, ORDER, AMR, 160>(a, entries);
    } else {
        return plan_march3d<R, ORDER, DIR, 128>(a, entries);
    }
}
// chip fills of the three sweeps together
template <class R, int ORDER, bool AMR> double sweep_waves(const Args3D &a0, unsigned entries)
{
    Args3D a = a0;
    return plan_sweep3d<R, ORDER, AMR, 0>(a, entries).waves + plan_sweep3d<R, ORDER, AMR, 1>(a, entries).waves +
           plan_sweep3d<R, ORDER, AMR, 2>(a, entries).waves;
}
// the sweep of direction DIR; max_smem: ask for the largest shared memory per SM
template <class R, int ORDER, bool AMR, int DIR, int OPT>
void launch_sweep3d(const Args3D &a0, unsigned entries, bool max_smem, cudaStream_t s)
{
    Args3D a = a0;
    const SweepPlan p = plan_sweep3d<R, ORDER, AMR, DIR>(a, entries);
    auto go = [&](void (*k)(Args3D)) {
        if (p.smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem);
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        at.val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
        cudaLaunchConfig_t c{};
        c.gridDim = p.grid;
        c.blockDim = dim3(p.threads);
        c.dynamicSmemBytes = p.smem;
        c.stream = s;
        c.attrs = &at;
        c.numAttrs = max_smem ? 1 : 0;
        cudaLaunchKernelEx(&c, k, a);
    };
    if constexpr (DIR == 0) {
        if constexpr (AMR)
            if (p.threads == 96) return go(sweepx3d_kernel<R, ORDER, AMR, OPT, 96>);
        go(sweepx3d_kernel<R, ORDER, AMR, OPT, 160>);
    } else {
        if constexpr (AMR)
            if (p.threads == 64) return go(march3d_kernel<R, ORDER, AMR, DIR, OPT, 64>);
        go(march3d_kernel<R, ORDER, AMR, DIR, OPT, 128>);
    }
}

} // namespace fxb
