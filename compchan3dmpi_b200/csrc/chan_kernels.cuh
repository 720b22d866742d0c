// chan_kernels.cuh -- sm_100a kernels of the compressible-channel time step.
//
// Device layout (all FP64):
//   Q  [5][nP3+2][nP2+2][px]   conservative state rho,rho*u,rho*v,rho*w,rho*E.
//                              Indices equal the reference's solV(0:nP1+1,
//                              0:nP2+1,0:nP3+1,1:5) (v1.10/codes/main_v1.9.f90:43).
//                              The 2-deep periodic ghosts in x are written by the
//                              stage kernel itself, those in y by the kernel after
//                              it, so every read is plain.
//   WP [2][8][nP2+2][px]       primitive state of the two wall planes k=1, k=nP3:
//                              rho,u,v,w,E,T,p,mu.  The wall pressure is a
//                              state variable of its own (pressure BC).
//   CS [nP3+2][4][7]           var at the four periodic corner columns.  The
//                              reference never refreshes these (its halo
//                              datatypes skip corners), yet its plane
//                              statistics sum them; kept only for that.
//
// One RK stage = k_stage (fluxes + update, fused) + k_wall (wall BC +
// pressure BC, and the ghost rows in y).  k_stats_part + k_stats_fin run every istat steps.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "chan_internal.h"
#include "phase_bits.h"

namespace chan {

// Step counter and time of the step being computed, kept on the device for
// launches replayed from a CUDA graph (whose kernel arguments are fixed at
// capture); k_clock_advance moves it at the start of every step.
struct DevClock {
    long long step;
    double time;
};

struct DevStatus {
    int blown;             // rho<0 or T<0 seen (reference blow-up test)
    int ijk[3];            // one offending point, 1-based reference indices
    int nonfinite;         // NaN/Inf seen
    int nf_ijk[3];
    long long blown_step;  // step in which the blow-up happened
    int stall;             // 1: a stage kernel's bulk copy did not complete in time; 2: misaligned staging area
    int pad;
};

// Boundary condition of one wall plane (plug-in of the reference's wall-BC
// variants in v1.9_strat, v1.9_groov, v1.9_groov_strat, v1.9_STWNV and v1.9_RD, lines ~605-640).
struct WallBC {
    int vel;              // 0 no-slip; 1 slip mask: c0*u1+c1*u2+c2*u3 = g where mask, else no-slip;
                          // 2 prescribed (u_w, v_w) field; 3 wave v_w = A sin(k x1 + om t + ph*(j odd))
    int therm;            // 0 isothermal Tw; 1 fixed one-sided gradient c0*T1+c1*T2+c2*T3 = dTdz
    double Tw, dTdz, g;
    double A, kx, om, ph;
    const unsigned char *mask;  // [nP2][nP1], 1-based (i,j) at (j-1)*nP1 + i-1
    const double *uv;           // [2][nP2][nP1]
    const double *x1;           // [nP1] x coordinates for the wave
};

// Flux arithmetic is templated on its real type R: double for the plain FP64
// path, float for the mixed-precision path (FP32 fluxes and stage storage,
// FP64 primitive recovery, RK accumulation and reductions).  FluxC holds the
// constants the flux formulas use, in R.
template <typename R>
struct FluxC {
    R invRe, ggM, two3rd, kq, inv_gM2;
    R hdx, hdy, sx8, sx12, sy8, sy12;
    R pex, pey, PexVal, PeyVal, pez_val;
};

struct KParams {
    // geometry
    int n1, n2, n3, px, NJ, kchunk;
    long long plane, vol;
    // state: stage input and output in the stage's storage type (double, or
    // float for the intermediate stages of the mixed-precision path); the RK
    // base state is always double
    const void *qin;
    const double *qbase;
    void *qout;
    double *wp;
    const double *cs;
    const double *czh;    // 0.5*invdXi*invJac(k), [nP3+2]
    // the stage kernel's constants of each plane (KTab), [nP3+2][8], in its ring type
    const void *ktab;
    // forcing / stats
    double *stat;         // stat1[7*n3] | stat2[7*n3] | corr[9*n3] | tau[2]
    double *tacc;         // running sums of the same 23*n3+2 numbers over statistics steps
    DevStatus *status;
    // physics
    double invRe, ggM, ggMh, gM2, inv_gM2, kq, two3rd;
    double hdx, hdy, sx8, sx12, sy8, sy12, invdx, invdy;
    double pex, pey, pez_val;   // Re*dx, Re*dy (x,y Peclet prefactors); PezVal
    double PexVal, PeyVal;
    double inv_dz1, inv_dzN;
    double Twb, Twt, muwb, muwt;
    FluxC<double> cd;     // flux constants in double (plain FP64 path)
    FluxC<float> cf;      // and in float (mixed-precision path)
    double f1[3], f2[3], b1[3], b2[3];  // wall one-sided coefficients
    // RK stage
    double rk_a, rk_b, rk_cdt;
    double rk_eps;        // a + b - 1 of the rounded a, b (0 but for a = 1/3, b = 2/3)
    int rk_mode;          // 0: in + cdt*R ; 1: base + cdt*R ; 2: a*base + b*in + cdt*R
    int check;            // last stage of a step: run the blow-up test
    int force_on;
    int acc_on;           // statistics steps also add into tacc (time averaging)
    int wall_custom;      // any wall uses a non-default WallBC
    WallBC wbc[2];
    // buoyancy body force ri*rho*(T - tref) on the wall-normal momentum and its
    // work ggM*w*(that) on the energy (a Boussinesq-style term for stratified
    // sweeps; the reference has none).  buoy_on = 0 leaves the RHS unchanged.
    double ri, tref;
    int buoy_on;
    double time;          // time of the step being computed (the reference's `time`)
    long long step;       // step number being computed
    const DevClock *clk;  // non-null in graph replays: step and time come from here
};

// step / time of the step being computed (kernel argument, or the device clock)
__device__ __forceinline__ long long kstep(const KParams &P) { return P.clk ? P.clk->step : P.step; }
__device__ __forceinline__ double ktime(const KParams &P) { return P.clk ? P.clk->time : P.time; }

__device__ __forceinline__ bool frozen(const DevStatus *st, long long step)
{
    // after a blow-up the reference stops; later steps do nothing here
    volatile const DevStatus *v = st;
    return v->blown && v->blown_step < step;
}

__device__ __forceinline__ void flag_blown(DevStatus *st, int i, int j, int k, long long step)
{
    if (atomicCAS(&st->blown, 0, 1) == 0) {
        st->ijk[0] = i; st->ijk[1] = j; st->ijk[2] = k;
        st->blown_step = step;
    }
}

__device__ __forceinline__ void flag_nonfinite(DevStatus *st, int i, int j, int k)
{
    if (atomicCAS(&st->nonfinite, 0, 1) == 0) {
        st->nf_ijk[0] = i; st->nf_ijk[1] = j; st->nf_ijk[2] = k;
    }
}

// Single-rounding multiply-add in the ring type.  The viscous fluxes are
// written with explicit FMAs so that every place that evaluates one (own
// columns, halo lanes, the k-march prologue) rounds it the same way, and a
// point's result does not depend on the launch shape that computed it.
template <typename R>
__device__ __forceinline__ R fmaR(R a, R b, R c);
template <>
__device__ __forceinline__ double fmaR<double>(double a, double b, double c) { return __fma_rn(a, b, c); }
template <>
__device__ __forceinline__ float fmaR<float>(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// an add the compiler may not fuse with a product feeding it
template <typename R>
__device__ __forceinline__ R addR(R a, R b);
template <>
__device__ __forceinline__ double addR<double>(double a, double b) { return __dadd_rn(a, b); }
template <>
__device__ __forceinline__ float addR<float>(float a, float b) { return __fadd_rn(a, b); }

// ---------------------------------------------------------------------------
// Inviscid stencil weights.  Both branches of the reference's hybrid scheme are
// linear in the conservative variable once the velocities are fixed, so a
// point's flux derivative along one axis is sum_m w[m]*Q(offset m-2) with
// weights shared by all five variables.
//  central : (-u2 Q2 + 8 u1 Q1 - 8 u-1 Q-1 + u-2 Q-2) /(12 d)   main_v1.9.f90:364-368
//  QUICK   : ue*Qe - uw*Qw, face values upwinded on the face velocity sign,
//            the four sign branches of main_v1.9.f90:335-361
template <typename R>
__device__ __forceinline__ void quick_weights(R um1, R u0, R up1, R s8, R w[5])
{
    const R r1 = (u0 + up1) * R(0.5);  // tmpR1, east face
    const R r2 = (u0 + um1) * R(0.5);  // tmpR2, west face
    const bool e = r1 >= R(0), f = r2 >= R(0);
    const R R1 = r1 * s8, R2 = r2 * s8;
    // east face value at offsets -1,0,+1,+2 ; west face at -2,-1,0,+1
    const R ae_m1 = e ? R(-1) : R(0), ae_0 = e ? R(6) : R(3), ae_1 = e ? R(3) : R(6), ae_2 = e ? R(0) : R(-1);
    const R bw_m2 = f ? R(-1) : R(0), bw_m1 = f ? R(6) : R(3), bw_0 = f ? R(3) : R(6), bw_1 = f ? R(0) : R(-1);
    w[0] = -R2 * bw_m2;
    w[1] = fmaR(R1, ae_m1, -(R2 * bw_m1));
    w[2] = fmaR(R1, ae_0, -(R2 * bw_0));
    w[3] = fmaR(R1, ae_1, -(R2 * bw_1));
    w[4] = R1 * ae_2;
}

// s12o: the outer pair's coefficient (s12, or 0 where the scheme next to a wall
// uses the inner pair alone)
template <typename R>
__device__ __forceinline__ void central_weights(R um2, R um1, R up1, R up2, R s12, R s12o, R w[5])
{
    w[0] = um2 * s12o;
    w[1] = R(-8) * um1 * s12;
    w[2] = R(0);
    w[3] = R(8) * up1 * s12;
    w[4] = -(up2 * s12o);
}

template <typename R>
__device__ __forceinline__ void inv_weights(R um2, R um1, R u0, R up1, R up2, bool quick, R s8, R s12, R s12o, R w[5])
{
    // Both weight sets, then a select per weight.  The switch differs from lane
    // to lane where the cell Peclet number crosses its limit, and a branch there
    // runs both paths one after the other (2.6% of the FP64 stage time, 1% of the
    // float one).
    R a[5], b[5];
    quick_weights(um1, u0, up1, s8, a);
    central_weights(um2, um1, up1, up2, s12, s12o, b);
#pragma unroll
    for (int m = 0; m < 5; m++) w[m] = quick ? a[m] : b[m];
}

// the first four terms of sum_m w[m] q[m], in the order of the offsets
template <typename R>
__device__ __forceinline__ R wsum4(const R w[5], R q0, R q1, R q2, R q3)
{
    return fmaR(w[3], q3, fmaR(w[2], q2, fmaR(w[0], q0, w[1] * q1)));
}
template <typename R>
__device__ __forceinline__ R wsum(const R w[5], R q0, R q1, R q2, R q3, R q4)
{
    return fmaR(w[4], q4, wsum4(w, q0, q1, q2, q3));
}

// ---------------------------------------------------------------------------
// Viscous / pressure flux vectors of main_v1.9.f90:457-538 in stress form.
// fD2..fD5 (fD1 = 0).  The energy component uses the identity
//   ggM*u*p + dissF = ggM*(u*fD2 + v*fD3 + w*fD4),
// which is the reference's dissF regrouped (same terms, different rounding).
template <typename R>
struct SlotT {
    const R *U, *V, *W, *T;
};

// pressure at box point b, rho*T/(gama*Ma^2) from the density RHO of the Q ring
// and T of the primitive ring (interior planes only)
template <typename R>
__device__ __forceinline__ R pres_at(const FluxC<R> &C, const SlotT<R> &s, const R *RHO, int b)
{
    return (RHO[b] * s.T[b]) * C.inv_gM2;
}

// fD from the gradients at one point: [p + 2/3 mu/Re div - 2 mu/Re u_x,
// -mu/Re (v_x+u_y), -mu/Re (w_x+u_z), -kq mu T_x + ggM (u fD2 + v fD3 + w fD4)]
template <typename R>
__device__ __forceinline__ void fd_point(const FluxC<R> &C, R mu, R pr, R u0, R v0, R w0, R ux, R vy, R wz, R vx,
                                         R uy, R wx, R uz, R Tx, R f[4])
{
    const R mr = mu * C.invRe, kqm = C.kq * mu;
    const R div = addR(addR(ux, vy), wz);
    const R pd = fmaR(C.two3rd * mr, div, pr);
    const R t12 = mr * addR(vx, uy);
    const R f2 = fmaR(-(R(2) * mr), ux, pd);
    const R f4 = -(mr * addR(wx, uz));
    f[0] = f2;
    f[1] = -t12;
    f[2] = f4;
    f[3] = fmaR(C.ggM, fmaR(w0, f4, fmaR(u0, f2, -(v0 * t12))), -(kqm * Tx));
}

// gD from the gradients at one point (gD2 = fD3, the shared shear stress)
template <typename R>
__device__ __forceinline__ void gd_point(const FluxC<R> &C, R mu, R pr, R u0, R v0, R w0, R ux, R vy, R wz, R vx,
                                         R uy, R wy, R vz, R Ty, R g[4])
{
    const R mr = mu * C.invRe, kqm = C.kq * mu;
    const R div = addR(addR(ux, vy), wz);
    const R pd = fmaR(C.two3rd * mr, div, pr);
    const R t12 = mr * addR(vx, uy);
    const R g3 = fmaR(-(R(2) * mr), vy, pd);
    const R g4 = -(mr * addR(wy, vz));
    g[0] = -t12;
    g[1] = g3;
    g[2] = g4;
    g[3] = fmaR(C.ggM, fmaR(w0, g4, fmaR(v0, g3, -(u0 * t12))), -(kqm * Ty));
}

// The flux helpers below take plane t's primitives from the ring slot s, plane
// t+1's from sp, and plane t-1's values at point b as scalars (um, vm, wm),
// which the caller keeps outside the ring.
template <int BX, typename R>
__device__ __forceinline__ void visc_fx(const FluxC<R> &C, const SlotT<R> &s, R um, R wm, const SlotT<R> &sp,
                                        const R *MU, const R *RHO, int b, R czt, R f[4])
{
    const R ux = (s.U[b + 1] - s.U[b - 1]) * C.hdx;
    const R uy = (s.U[b + BX] - s.U[b - BX]) * C.hdy;
    const R vx = (s.V[b + 1] - s.V[b - 1]) * C.hdx;
    const R vy = (s.V[b + BX] - s.V[b - BX]) * C.hdy;
    const R wx = (s.W[b + 1] - s.W[b - 1]) * C.hdx;
    const R Tx = (s.T[b + 1] - s.T[b - 1]) * C.hdx;
    const R uz = (sp.U[b] - um) * czt;
    const R wz = (sp.W[b] - wm) * czt;
    fd_point(C, MU[b], pres_at(C, s, RHO, b), s.U[b], s.V[b], s.W[b], ux, vy, wz, vx, uy, wx, uz, Tx, f);
}

template <int BX, typename R>
__device__ __forceinline__ void visc_fy(const FluxC<R> &C, const SlotT<R> &s, R vm, R wm, const SlotT<R> &sp,
                                        const R *MU, const R *RHO, int b, R czt, R g[4])
{
    const R ux = (s.U[b + 1] - s.U[b - 1]) * C.hdx;
    const R uy = (s.U[b + BX] - s.U[b - BX]) * C.hdy;
    const R vx = (s.V[b + 1] - s.V[b - 1]) * C.hdx;
    const R vy = (s.V[b + BX] - s.V[b - BX]) * C.hdy;
    const R wy = (s.W[b + BX] - s.W[b - BX]) * C.hdy;
    const R Ty = (s.T[b + BX] - s.T[b - BX]) * C.hdy;
    const R vz = (sp.V[b] - vm) * czt;
    const R wz = (sp.W[b] - wm) * czt;
    gd_point(C, MU[b], pres_at(C, s, RHO, b), s.U[b], s.V[b], s.W[b], ux, vy, wz, vx, uy, wy, vz, Ty, g);
}

template <typename R>
__device__ __forceinline__ void visc_fz_vals(const FluxC<R> &C, R ux, R vy, R wx, R wy, R u, R v, R w, R mu, R pr,
                                             R uz, R vz, R wz, R Tz, R h[4])
{
    const R mr = mu * C.invRe, kqm = C.kq * mu;
    const R div = addR(addR(ux, vy), wz);
    const R h2 = -(mr * addR(wx, uz));
    const R h3 = -(mr * addR(wy, vz));
    const R h4 = fmaR(-(R(2) * mr), wz, fmaR(C.two3rd * mr, div, pr));
    h[0] = h2;
    h[1] = h3;
    h[2] = h4;
    h[3] = fmaR(C.ggM, fmaR(w, h4, fmaR(v, h3, u * h2)), -(kqm * Tz));
}

// periodic image of index i in 0..n+1 (duplicate-point period n-2):
// q(0)=q(n-2), q(1)=q(n-1), q(n)=q(2), q(n+1)=q(3)
__device__ __forceinline__ int wrap_idx(int i, int n)
{
    if (i == 0) return n - 2;
    if (i == 1) return n - 1;
    if (i == n) return 2;
    if (i == n + 1) return 3;
    return i;
}

// ---------------------------------------------------------------------------
// Short math for the transport law mu = k = T^0.7 (main_v1.9.f90:643, 720) and
// for 1/rho.  Both start from hardware approximations and refine in FP64.
//
// The seeds are the approximations themselves: rcp.approx.ftz.f64 for the
// reciprocal, ex2.approx.ftz.f32 after lg2.approx.ftz.f32 for the power.  The FP64
// refinement squares (Newton) or cubes (Halley) the seed's relative error at
// each step, so it reaches the same accuracy from them as from exact float
// values.  Measured against the alternatives on the FP64 stage kernel: the
// correctly rounded float reciprocal __frcp_rn and the library exp2f
// (CHAN_EXACT_SEEDS) 7.5% slower; the float reciprocal approximation with its
// two conversions (CHAN_F32_RCP_SEED) 1.2% slower.
__device__ __forceinline__ float seed_rcp(float x)
{
#ifndef CHAN_EXACT_SEEDS
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return __frcp_rn(x);
#endif
}
__device__ __forceinline__ float seed_log2(float x)
{
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float seed_exp2(float x)
{
#ifndef CHAN_EXACT_SEEDS
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return exp2f(x);
#endif
}

// rcp_fast: 1/x from the seed r by one third-order step, r (1 + e + e^2) with
// e = 1 - x r (the seed's error cubed: to about 1 ulp), one dependent FMA fewer
// than two Newton steps (CHAN_RCP_NEWTON2; 0.5% of the FP64 stage time).  Valid
// for |x| in the normal range, which covers rho and mu of any physical state.
__device__ __forceinline__ double rcp_fast(double x)
{
#if !defined(CHAN_F32_RCP_SEED) && !defined(CHAN_EXACT_SEEDS)
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
#else
    double r = (double)seed_rcp((float)x);
#endif
#ifndef CHAN_RCP_NEWTON2
    // one step of third order: 1/x = r / (1 - e) = r (1 + e + e^2 + ...), e = 1 - x r
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
#else
    double e = fma(-x, r, 1.0);
    r = fma(r, e, r);
    e = fma(-x, r, 1.0);
    return fma(r, e, r);
#endif
}

// pow07: y = T^0.7 = T x with x = T^-0.3, the positive root of x^10 T^3 = 1.
// From the float seed x0 = exp2(-0.3 log2 T) (relative error ~3e-7),
// e = 1 - x0^10 T^3 (~3e-6) and x = x0 (1 - e)^(-1/10), whose binomial series
// 1 + e/10 + 0.055 e^2 + ... is cut after e^2 (the rest ~1e-18): twelve FP64
// operations and no division, so the result is limited by FP64 rounding
// (~2 ulp).  The earlier form, one Halley step on y^10 = T^7 with a reciprocal
// (CHAN_POW_HALLEY), takes 0.4% more of the FP64 stage time.  T <= 0 gives NaN
// (the reference's T**0.7 does for T < 0; T = 0 does not arise).
__device__ __forceinline__ double pow07(double T)
{
#ifndef CHAN_POW_HALLEY
    // y = T * x with x = T^-0.3, the root of x^10 T^3 = 1.  From the float seed
    // x0 (relative error ~3e-7), e = 1 - x0^10 T^3 and
    // x = x0 (1 - e)^(-1/10) = x0 (1 + e/10 + 0.055 e^2 + 0.0385 e^3 + ...):
    // the series to e^2 leaves ~1e-18; no division.
    const double x0 = (double)seed_exp2(-0.3f * seed_log2((float)T));
    const double t2 = T * T, t3 = t2 * T;
    const double x2 = x0 * x0, x4 = x2 * x2, x8 = x4 * x4, x10 = x8 * x2;
    const double e = fma(-x10, t3, 1.0);
    const double pe = fma(fma(0.0385, e, 0.055), e, 0.1);
    return T * fma(x0 * e, pe, x0);
#else
    const float tf = (float)T;
    double y = (double)seed_exp2(0.7f * seed_log2(tf));
    const double T2 = T * T, T4 = T2 * T2, a = (T4 * T2) * T;
    const double y2 = y * y, y4 = y2 * y2, y8 = y4 * y4, u = y8 * y2;
    const double num = fma(9.0, u, 11.0 * a);
    const double den = fma(11.0, u, 9.0 * a);
    return (y * num) * rcp_fast(den);
#endif
}

// primitives of one point from the conservative state (calcPrim, main_v1.9.f90:600-609)
__device__ __forceinline__ void prims_from_q(const KParams &P, const double q[5], double &u, double &v,
                                             double &w, double &T)
{
    const double r = rcp_fast(q[0]);
    u = q[1] * r;
    v = q[2] * r;
    w = q[3] * r;
    const double E = q[4] * r;
    // explicit FMAs: the same bits wherever a point's primitives are formed
    T = __fma_rn(-P.ggMh, __fma_rn(w, w, __fma_rn(v, v, u * u)), E);
}

// ---------------------------------------------------------------------------
// The fused stage kernel.
//
// A CTA owns a TI x TJ tile of interior (i,j) columns and marches a chunk of
// interior planes k = kb..ke.  A thread owns one x column (FP64) or two neighbouring
// ones (float: i even, so that every access of its pair, of its y neighbours and of its
// x stencil is an aligned 8-byte one in shared, 16-byte one in global memory).
// Bound by instruction issue and latency, not by HBM: 256x193x192, a launch, FP64 0.604 ->
// 0.505 ms and mixed 0.441 -> 0.346 ms with the plane's scattered per-thread loads (RK
// base, tables, forcing density) by bulk copies, the wall-normal sum completed one plane
// behind, the x images under one branch and the y images left to the wall launch.
// Shared memory holds, for the tile plus a 2-point halo box
// ((TI+4) x (TJ+4)):
//   Q (5 vars)      of planes t, t+1, t+2   (3-slot ring; t+2 in flight)
//   prims u,v,w,T   of planes t, t+1        (2-slot ring)
//   mu              of planes t, t+1        (2-slot ring; p is rho T / (gama Ma^2))
//   fD, gD          of plane t on the tile plus a 1-point halo
// Plane t-1 is kept where it is still read: each thread's own columns (Q, u,
// v, w, T) in registers, and the halo points of the halo-flux lanes in a small
// shared array.  Each thread also keeps its own columns' Q and w at t-2, hD at
// t-1 and the unfinished sums of plane t-1 in registers.
//
// The Q box of each plane arrives by one tiled bulk tensor copy (TMA) issued
// about two thirds of a plane ahead by one thread and completed on an mbarrier,
// so Q is read from DRAM once per stage with no per-thread load instructions;
// the halo re-reads of neighbouring CTAs come from L2.  Each staged box point is
// then converted to primitives once per CTA.  The stage whose input is stored in
// a wider type than the ring (the first stage of the mixed-precision path, double
// in, float rings) loads its boxes with per-thread loads instead.
//
// A plane takes two CTA barriers: after the box conversion (with which the
// inviscid x/y sums of the plane share one straight-line block) and after the
// viscous fluxes.  None ends the plane, so
// warps that finish the update early go on into the next plane's loads and
// conversion while the others complete theirs.
//
// Types: QI / QO are the storage types of the stage's input and output state,
// R the type of the shared rings and of the flux arithmetic.  The plain FP64
// path is <double, double, double>.  The mixed-precision path stores the
// intermediate stage states in float and evaluates the fluxes in float; the
// primitive recovery (T from the total energy), the RK update against the
// double base state, the forcing and the blow-up test stay in double.
// constants of plane k: 0.5*invdXi*invJac; invdXi*invJac/8 (QUICK); the central
// scheme's factor of the inner and of the outer pair, invdXi*invJac/12 both, but
// next to a wall, where the scheme is the second-order (-w(k-1), 0, w(k+1)) * czh,
// czh/8 and 0; Re*dXi*jac (the Peclet factor), -infinity next to a wall, so that the
// switch never picks QUICK there.
enum KTab { kCzh = 0, kS8 = 1, kS12 = 2, kS12o = 3, kPez = 4, kTabWords = 8 };

template <int TI, int TJ, typename R>
struct StageShape {
    // NT threads of PX neighbouring x points each, TX per row of the tile.  Two points
    // share their loads, addresses and loop overhead (32% fewer instructions), but
    // need twice the registers: that pays in float (0.344 against 0.398 ms per launch at
    // 256x193x192 with one point, in 80 registers); in FP64 two points of 255 registers
    // leave two warps per scheduler (0.718 against 0.502 ms).
    static constexpr int PX = sizeof(R) == 4 ? 2 : 1;
    static constexpr int BX = TI + 4, BY = TJ + 4, NB = BX * BY, TX = TI / PX, NT = TX * TJ;
    // fD rows: [left halo, TI own points, right halo], padded so that own pairs are
    // aligned; own points from FO on.  fD3 = gD2 is one array with both halos.
    static constexpr int FO = PX, FP = TI + 2 * FO;
    static constexpr int NFX = TJ * FP, NGY = (TJ + 2) * TI, NXY = (TJ + 2) * FP;
    // one Q slot: the 5-variable box of one plane, rounded up to 128 bytes
    // (the alignment of a bulk tensor copy's shared-memory destination)
    static constexpr size_t box_bytes = (size_t)5 * NB * sizeof(R);
    static constexpr size_t qslot_bytes = (box_bytes + 127) / 128 * 128;
    static constexpr int QSLOT = (int)(qslot_bytes / sizeof(R));     // slot stride in R elements
    static constexpr size_t q_bytes = 3 * qslot_bytes;
    static constexpr int pr_words = 2 * 4 * NB;
    static constexpr int mu_words = 2 * NB;
    static constexpr int fg_words = 3 * NFX + 3 * NGY + NXY;
    // the tile's RK base of one plane (double), by bulk tensor copy: 128-byte aligned
    static constexpr size_t base_off = (q_bytes + sizeof(R) * (size_t)(pr_words + mu_words + fg_words) + 127) / 128 * 128;
    static constexpr size_t base_bytes = sizeof(double) * 5 * TI * TJ;
    // per plane (4 slots): its constants (KTab) and 16 bytes of the forcing's density
    static constexpr size_t tab_off = base_off + base_bytes;
    static constexpr size_t tab_bytes = kTabWords * sizeof(R), rb_off = tab_off + 4 * tab_bytes;
    // plane t-1 values (u or v, and w) of the halo-flux points: 2*TJ of the two
    // x-halo columns, then 2*TI of the two y-halo rows
    static constexpr int NHL = 2 * TJ + 2 * TI;
    static constexpr size_t hl_off = rb_off + 4 * 16;
    static constexpr size_t bar_off = (hl_off + sizeof(R) * 2 * (size_t)NHL + 7) / 8 * 8;
    static constexpr size_t bytes = bar_off + 5 * sizeof(unsigned long long) + 2 * sizeof(int);
    // resident CTAs per SM the register budget is sized for: as many as the
    // 228 KB of shared memory per SM hold (1 KB of it reserved per CTA), and
    // never fewer registers than a thread needs (one point in double, two in float)
    static constexpr int MINR = 128;
    static constexpr int minb_smem = (int)(233472 / (bytes + 1024));
    static constexpr int minb_regs = 65536 / (MINR * NT);
    static constexpr int minb = minb_regs < minb_smem ? minb_regs : minb_smem;
};

template <typename R>
__device__ __forceinline__ const FluxC<R> &fluxc(const KParams &P);
template <>
__device__ __forceinline__ const FluxC<double> &fluxc<double>(const KParams &P) { return P.cd; }
template <>
__device__ __forceinline__ const FluxC<float> &fluxc<float>(const KParams &P) { return P.cf; }

// mu = T^0.7 in the ring type: pow07 in double; exp2(0.7 log2 T) in float
template <typename R>
__device__ __forceinline__ R mu_of(double T);
template <>
__device__ __forceinline__ double mu_of<double>(double T) { return pow07(T); }
template <>
__device__ __forceinline__ float mu_of<float>(double T)
{
    // the hardware log2 and exp2 approximations (relative error about 2^-21, well
    // inside the float path's own rounding); the library log2f/exp2f cost 2.5% of
    // the float stage kernel
    return seed_exp2(0.7f * seed_log2((float)T));
}

// PX neighbouring elements in one access (the address is a multiple of its size)
template <typename T>
struct Pair;
template <>
struct Pair<double> { using V = double2; };
template <>
struct Pair<float> { using V = float2; };
template <int PX, typename T, typename R>
__device__ __forceinline__ void ldp(const T *p, R out[PX])
{
    if constexpr (PX == 2) {
        const typename Pair<T>::V v = *reinterpret_cast<const typename Pair<T>::V *>(p);
        out[0] = (R)v.x;
        out[1] = (R)v.y;
    } else {
        out[0] = (R)*p;
    }
}
template <int PX, typename T, typename R>
__device__ __forceinline__ void stp(T *p, const R in[PX])
{
    if constexpr (PX == 2) {
        typename Pair<T>::V v;
        v.x = (T)in[0];
        v.y = (T)in[1];
        *reinterpret_cast<typename Pair<T>::V *>(p) = v;
    } else {
        *p = (T)in[0];
    }
}
// the same from global memory, as doubles.  Plain loads, never the read-only path: an
// early-launched CTA is resident while the kernel before it still writes this state (in
// the persistent ensemble kernel, other CTAs of the same launch do).
template <int PX, typename T>
__device__ __forceinline__ void ldgp(const T *p, double out[PX])
{
    if constexpr (PX == 2) {
        const typename Pair<T>::V v = *reinterpret_cast<const typename Pair<T>::V *>(p);
        out[0] = (double)v.x;
        out[1] = (double)v.y;
    } else {
        out[0] = (double)*p;
    }
}


// asynchronous global->shared copy of PX doubles (no register staging)
template <int PX>
__device__ __forceinline__ void cp_async_d(double *dst, const double *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (PX == 2) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ---- tiled bulk tensor copies into this CTA's shared memory, with mbarriers
__device__ __forceinline__ unsigned smem_u32addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init_one(unsigned long long *bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32addr(bar)) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// order the CTA's earlier generic-proxy accesses of shared memory (made
// visible to this thread by a CTA barrier) before its later async-proxy writes
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// one arrival on the barrier, which then waits for `bytes` of copies
__device__ __forceinline__ void mbar_expect(unsigned long long *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32addr(bar)), "r"(bytes)
                 : "memory");
}
// `bytes` (a multiple of 16) from global memory at src (16-byte aligned) into dst
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32addr(bar))
        : "memory");
}
// the 4-D box at (x, y, z, w) of the tensor map into dst.  No multicast: the box
// lands in this CTA's shared memory only.
__device__ __forceinline__ void tma_load_box(void *dst, const CUtensorMap *map, int x, int y, int z, int w,
                                             unsigned long long *bar)
{
    const unsigned b = smem_u32addr(bar);
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];" ::"r"(smem_u32addr(dst)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(b)
        : "memory");
}

__device__ __forceinline__ bool mbar_try(unsigned a, unsigned parity)
{
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    return done != 0;
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// wait for phase `parity` of the barrier; false when about a second passed
// without it (the caller records the error and stops)
constexpr unsigned long long kCopyWaitNs = 1000000000ull;
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long *bar, unsigned parity)
{
    const unsigned a = smem_u32addr(bar);
    if (mbar_try(a, parity)) return true;
    const unsigned long long t0 = global_ns();
    while (!mbar_try(a, parity))
        if (global_ns() - t0 > kCopyWaitNs) return false;
    return true;
}

// One CTA's work of the stage kernel on tile (bx, by) and k-chunk bz, for
// thread (tx, ty).  BUOYM: 0 no buoyancy term, 1 with it, 2 as P.buoy_on
// says.  PERSIST: called from the persistent ensemble kernel, where the state
// was written earlier in the same launch: a proxy fence before the first box copy; *stuck
// is set when the CTA must not use its shared memory again.
template <int TI, int TJ, typename QI, typename QO, typename R, int BUOYM, bool PERSIST>
__device__ __forceinline__ void stage_body(const KParams &P, const CUtensorMap *tmq, const CUtensorMap *tmb, int bx, int by,
                                           int bz, int tx, int ty, unsigned char *smem_raw, int *stuck)
{
    using S = StageShape<TI, TJ, R>;
    using Slot = SlotT<R>;
    constexpr int BX = S::BX, NB = S::NB, NT = S::NT, QSLOT = S::QSLOT, FP = S::FP, PX = S::PX;
    constexpr int FO = S::FO, NHL = S::NHL;
    // FP64: the wall-normal terms are folded into the carried sum as they come;
    // the float kernels keep the order of the one-pass sum
    constexpr bool FOLD = sizeof(R) == 8;
    // boxes by bulk tensor copy when the input is stored in the ring type
    constexpr bool TMA = std::is_same<QI, R>::value;
    static_assert(TI % PX == 0 && 2 * TJ <= 32 && NT >= 32, "tile layout");
    R *sQ = reinterpret_cast<R *>(smem_raw);                       // [3 slots][5][NB]
    R *sPr = reinterpret_cast<R *>(smem_raw + S::q_bytes);         // [2][4][NB] u,v,w,T
    R *sMU = sPr + S::pr_words;                                    // [2][NB] mu
    R *sF = sMU + S::mu_words;                                     // fD2, fD4, fD5 [3][TJ][FP], own points from FO on
    R *sG = sF + 3 * S::NFX;                                       // gD3, gD4, gD5 [3][TJ+2][TI]
    R *sX = sG + 3 * S::NGY;                                       // fD3 = gD2 [TJ+2][FP]
    double *sQB = reinterpret_cast<double *>(smem_raw + S::base_off);   // [5][TJ][TI]
    R *sT = reinterpret_cast<R *>(smem_raw + S::tab_off);               // [4][kTabWords]
    double *sRB = reinterpret_cast<double *>(smem_raw + S::rb_off);     // [4][2]
    R *sH = reinterpret_cast<R *>(smem_raw + S::hl_off);                // [2][NHL]
    // bar_off is a multiple of 8: the mask only keeps the compiler from folding the barriers'
    // addresses into registers of their own (without it the FP64 32x8 kernel spills 56 + 88
    // bytes instead of 12 + 12)
    unsigned long long *bar = reinterpret_cast<unsigned long long *>(reinterpret_cast<size_t>(smem_raw + S::bar_off) & ~(size_t)7);   // [4]: Q slots, RK base
    double *stau = reinterpret_cast<double *>(bar + 4);   // tauL - tauU
    int *sflag = reinterpret_cast<int *>(bar + 5);   // [0] the CTA leaves at once, [1] copies in flight
    const FluxC<R> &C = fluxc<R>(P);
    // the state pointers are read from the parameter space at each use: held
    // in registers across the kernel they cost spills
    auto qin = [&]() { return static_cast<const QI *>(P.qin); };
    auto qout = [&]() { return static_cast<QO *>(P.qout); };

    const bool buoy = BUOYM == 2 ? P.buoy_on != 0 : BUOYM == 1;
    const int tid = ty * S::TX + tx;
    if (tid == 0) {
        sflag[0] = frozen(P.status, kstep(P)) ? 1 : 0;
        sflag[1] = 0;
        // state written by other CTAs of this launch, read next by box copies
        if (PERSIST) asm volatile("fence.proxy.async.global;" ::: "memory");
        // a bulk copy needs a 128-byte aligned destination
        if (smem_u32addr(smem_raw) & 127u) {
            sflag[0] = 1;
            atomicExch(&P.status->stall, 2);
        }
        for (int s = 0; s < 4; s++) mbar_init_one(&bar[s]);
        fence_mbar_init();
        *stau = P.stat[23 * P.n3 + 0] - P.stat[23 * P.n3 + 1];
    }
    __syncthreads();
    if (sflag[0]) return;

    const int i0 = 2 + bx * TI, j0 = 2 + by * TJ;
    const int kb = 2 + bz * P.kchunk;
    const int ke = min(kb + P.kchunk - 1, P.n3 - 1);
    if (kb > ke) return;
    const int n1 = P.n1, n2 = P.n2, n3 = P.n3;
    const int i = i0 + PX * tx, j = j0 + ty;
    // the pair is loaded and its fluxes formed when its first point is a stored
    // one: the row pitch px >= nP1+2 is even, so the pair lies inside the row
    const bool col_ok = (i <= n1) && (j <= n2);
    const bool out0 = (i <= n1 - 1) && (j <= n2 - 1), out1 = (i + PX - 1 <= n1 - 1) && (j <= n2 - 1);
    const int bc = (ty + 2) * BX + PX * tx + 2;
    // offset of the own points' periodic image in x (0: none; the points of a pair that
    // have one have the same)
    const int xim = i <= 3 ? n1 - 2 : (i + PX - 1 >= n1 - 2 ? 2 - n1 : 0);
    const long long vol = P.vol, plane = P.plane;
    const long long colo = (long long)j * P.px + i;

    // ring slots by role, rotated once per plane: Q slots (indices 0..2) of
    // planes t, t+1, t+2; prims offsets of t, t+1; mu offsets of t, t+1
    int iZ = 1, iP = 2, iN = 0;
    int pZ = 0, pP = 4 * NB, mZ = 0, mP = NB;
    PhaseBits ph;   // of the next wait, per barrier
    auto slot = [&](int o) -> Slot {
        return Slot{sPr + o, sPr + o + NB, sPr + o + 2 * NB, sPr + o + 3 * NB};
    };
    auto smu = [&](int o) { return sMU + o; };
    auto sq = [&](int s, int v) { return sQ + s * QSLOT + v * NB; };
    // plane k's constants and forcing density, staged with its box
    auto ktab = [&](int which, int k) { return sT[(k & 3) * kTabWords + which]; };
    auto rbar = [&](int k) { return sRB[(k & 3) * 2 + ((k - 1) & 1)]; };

    // plane m's Q box into Q slot s, with the plane's constants and forcing density
    // (one thread; bulk copies).  Everything a plane reads per thread then comes from
    // shared memory: as plain loads, L1 hits most of them, the constants, the density
    // and the RK base below held up the warps for 18% of the FP64 stage time.
    auto issue = [&](int m, int s) {
        if (tid == 0) {
            fence_proxy_async_smem();
            mbar_expect(&bar[s], (unsigned)((TMA ? S::box_bytes : 0) + S::tab_bytes + 16));
            if (TMA) tma_load_box(sq(s, 0), tmq, i0 - 2, j0 - 2, m, 0, &bar[s]);
            bulk_load(sT + (m & 3) * kTabWords, static_cast<const R *>(P.ktab) + (size_t)m * kTabWords,
                      (unsigned)S::tab_bytes, &bar[s]);
            bulk_load(sRB + (m & 3) * 2, P.stat + ((m - 1) & ~1), 16u, &bar[s]);
            sflag[1] |= 1 << s;
        }
    };
    // the mixed path's first stage never has a base, its others always do
    const bool need_base = FOLD ? P.rk_mode != 0 : TMA;
    constexpr bool CHK = std::is_same<QO, double>::value;   // a step's last stage may be this kernel
    // FP64: the tile's RK base of plane m into its slot (barrier 3)
    auto issue_base = [&](int m) {
        if (FOLD && need_base && tid == 0) {
            fence_proxy_async_smem();
            mbar_expect(&bar[3], (unsigned)S::base_bytes);
            tma_load_box(sQB, tmb, i0, j0, m, 0, &bar[3]);
            sflag[1] |= 1 << 3;
        }
    };
    // wait for barrier s; false if its copies did not complete in time
    auto wait_slot = [&](int s) -> bool {
        const bool ok = mbar_wait_bounded(&bar[s], ph.next(s));
        ph.waited(s);
        if (ok && tid == 0) sflag[1] &= ~(1 << s);
        return ok;
    };
    // after a timed-out copy: record it and give every copy still in flight one more bounded
    // wait, so that none lands after the CTA has left its shared memory; if one still may, a
    // CTA of the persistent kernel takes up no other unit (*stuck).  waited: the slots whose
    // latest copy has been waited for.
    auto give_up = [&](int waited) {
        if (!FOLD) cp_async_wait<0>();
        if (tid == 0) {
            atomicExch(&P.status->stall, 1);
            for (int s = 0; s < 4; s++)
                if (sflag[1] & (1 << s)) {
                    if (!mbar_wait_bounded(&bar[s], ph.open(s, (waited >> s) & 1)) && PERSIST) *stuck = 1;
                }
        }
    };

    // own columns, carried from plane to plane: Q at t-1 and t-2, u, v, w, T at
    // t-1, w at t-2, hD at t-1; and what is known of plane t-1's update, which only
    // lacks what plane t+1 brings: Fs (FP64: the RK increment on Q; float rings: the
    // flux derivatives in x and y), its wall-normal switch (qk) and the QUICK weight of
    // Q(t+1) (w4).  Float rings add the wall-normal terms in the order of the one-pass
    // sum and carry them apart (H1p: that sum but its last term, hm: hD(t-2)).
    R qm2[5][PX], qm1[5][PX], Fs[PX][5], h1[PX][4], hm[PX][4], H1p[PX][5], w4[PX];
    R wm2[PX], um1[PX], vm1[PX], wm1[PX], Tm1[PX];
    bool qk[PX] = {}, qz[PX] = {};   // the wall-normal switch of planes t-1 and t
#pragma unroll
    for (int a = 0; a < PX; a++) {
#pragma unroll
        for (int c = 0; c < 5; c++) qm2[c][a] = qm1[c][a] = Fs[a][c] = H1p[a][c] = R(0);
#pragma unroll
        for (int c = 0; c < 4; c++) h1[a][c] = hm[a][c] = R(0);
        wm2[a] = um1[a] = vm1[a] = wm1[a] = Tm1[a] = w4[a] = R(0);
    }
    // box pairs this thread converts: the same columns for every plane
    // lp: box index of the pair's first point, -1 if that is outside the array
    // (its second point may be one past the array: converted from the copy's zero
    // fill or from the row's padding, stored, and read by no one).  lo: column offset.
    constexpr int NL = (NB / PX + NT - 1) / NT;
    int lp[NL];
    int lo[NL];
#pragma unroll
    for (int l = 0; l < NL; l++) {
        const int p = PX * (tid + l * NT);
        const int bj = p / BX, bi = p - bj * BX;
        const int gi = i0 - 2 + bi, gj = j0 - 2 + bj;
        lp[l] = p < NB && gi <= n1 + 1 && gj <= n2 + 1 ? p : -1;
        lo[l] = gj * P.px + gi;
    }

    // The inviscid x and y flux derivatives of plane t (F1 + G1) need only plane
    // t's Q box and u, v, which the previous plane converted: they are formed in
    // phase A, in the same straight-line block as the conversion of plane t+1's
    // box, whose dependency chains (reciprocal, power) they fill (1.7% of the
    // FP64 stage time, 2.4% of the float one, against forming them in phase E).
    // a row of the x stencil: PX + 4 values around the own points
    auto row = [&](const R *f, R x[PX + 4]) {
        if constexpr (PX == 2) {
            ldp<2>(f - 2, x);
            ldp<2>(f, x + 2);
            ldp<2>(f + 2, x + 4);
        } else {
#pragma unroll
            for (int m = 0; m < 5; m++) x[m] = f[m - 2];
        }
    };
    // FP64: what it leaves is W = a*(Qbase - Q) - cdt*(F1 + G1 + the wall-normal terms
    // of Q(t-2) and hD(t-1)), the part known so far of the RK update's increment on Q
    // (a*Qbase + b*Q = Q + a*(Qbase - Q) + eps*Q, eps = a + b - 1 the rounding of a and
    // b; the increment is small beside Q, so only its addition rounds at Q's size).  The base is thus read
    // here and not carried, and Q(t-2), hD(t-1) and w(t-2) end here, before the viscous
    // fluxes, where most values are live.
    auto inv_xy = [&](int t, R Fxy[PX][5]) {
        R mu0[PX], m0[PX], w[PX][5];
        const R *U = sPr + pZ + bc, *V = sPr + pZ + NB + bc;
        ldp<PX>(smu(mZ) + bc, mu0);
        {
            R x[PX + 4];
            row(U, x);
            ldp<PX>(sq(iZ, 1) + bc, m0);
#pragma unroll
            for (int a = 0; a < PX; a++) {
                const bool q = (C.pex * fabs(m0[a])) > C.PexVal * mu0[a];
                inv_weights(x[a], x[a + 1], x[a + 2], x[a + 3], x[a + 4], q, C.sx8, C.sx12, C.sx12, w[a]);
            }
#pragma unroll
            for (int c = 0; c < 5; c++) {
                row(sq(iZ, c) + bc, x);
#pragma unroll
                for (int a = 0; a < PX; a++) Fxy[a][c] = wsum(w[a], x[a], x[a + 1], x[a + 2], x[a + 3], x[a + 4]);
            }
        }
        {
            R y[5][PX];
#pragma unroll
            for (int m = 0; m < 5; m++) ldp<PX>(V + (m - 2) * BX, y[m]);
            ldp<PX>(sq(iZ, 2) + bc, m0);
            R wz[PX], cz = R(0);
            if constexpr (FOLD) {
                R w0[PX], m3[PX];
                ldp<PX>(sPr + pZ + 2 * NB + bc, w0);
                ldp<PX>(sq(iZ, 3) + bc, m3);
                const R pez = ktab(kPez, t), s8 = ktab(kS8, t), s12o = ktab(kS12o, t);
                cz = ktab(kCzh, t);
#pragma unroll
                for (int a = 0; a < PX; a++) {
                    qz[a] = (pez * fabs(m3[a])) > C.pez_val * mu0[a];
                    const R r2 = ((w0[a] + wm1[a]) * R(0.5)) * s8;   // weight of Q(t-2), as inv_weights has it
                    wz[a] = qz[a] ? (r2 >= R(0) ? r2 : R(0)) : wm2[a] * s12o;
                }
            }
#pragma unroll
            for (int a = 0; a < PX; a++) {
                const bool q = (C.pey * fabs(m0[a])) > C.PeyVal * mu0[a];
                inv_weights(y[0][a], y[1][a], y[2][a], y[3][a], y[4][a], q, C.sy8, C.sy12, C.sy12, w[a]);
            }
#pragma unroll
            for (int c = 0; c < 5; c++) {
                const R *Q = sq(iZ, c) + bc;
#pragma unroll
                for (int m = 0; m < 5; m++) ldp<PX>(Q + (m - 2) * BX, y[m]);
#pragma unroll
                for (int a = 0; a < PX; a++)
                    Fxy[a][c] = Fxy[a][c] + wsum(w[a], y[0][a], y[1][a], y[2][a], y[3][a], y[4][a]);
                if constexpr (FOLD) {
                    R qb[PX];
#pragma unroll
                    for (int a = 0; a < PX; a++) {
                        qb[a] = y[2][a];
                        Fxy[a][c] = fmaR(wz[a], qm2[c][a], Fxy[a][c]);
                        if (c > 0) Fxy[a][c] = fmaR(-h1[a][c > 0 ? c - 1 : 0], cz, Fxy[a][c]);
                    }
                    if (need_base) ldp<PX>(sQB + (c * TJ + ty) * TI + PX * tx, qb);
#pragma unroll
                    for (int a = 0; a < PX; a++)
                        Fxy[a][c] = fmaR(-(R)P.rk_cdt, Fxy[a][c], fmaR((R)P.rk_eps, y[2][a], (R)P.rk_a * (qb[a] - y[2][a])));
                }
            }
        }
    };

    // primitives, mu and p of plane m over the box, from its Q box in slot s (with
    // per-thread loads, Q is first loaded into the slot).  A wall plane's box
    // holds, at periodic duplicates and ghosts, the values of their image points:
    // the viscous fluxes next to a wall read the wall only there, and the
    // reference's flux at a duplicate column or row is the exchanged flux of its
    // image (whose wall values may differ from the duplicate's own under a
    // non-periodic wall BC).  hD on a wall plane reads the wall's own values from
    // memory instead (hflux_wall).
    auto convert = [&](int m, int s, int po, int mo, bool with_xy, R (*Fxy)[PX][5] = nullptr) {
        const Slot sl = slot(po);
        R *MU = smu(mo);
        const bool wall = (m == 1 || m == n3);
        const double *W = P.wp + (size_t)(m == 1 ? 0 : 8) * plane;
        auto one = [&](int l, bool wall_plane) {
            if (lp[l] < 0) return;
            const int p = lp[l];
            double q[5][PX];
            if (!TMA) {
                const long long off = (long long)m * plane + lo[l];
#pragma unroll
                for (int v = 0; v < 5; v++) {
                    ldgp<PX>(qin() + v * vol + off, q[v]);
                    stp<PX>(sq(s, v) + p, q[v]);
                }
            }
            double u[PX], vv[PX], w[PX], T[PX];
            R mu[PX];
            if (wall_plane) {
                const int bj = p / BX, bi = p - bj * BX;
                const long long wj = (long long)wrap_idx(j0 - 2 + bj, n2) * P.px;
#pragma unroll
                for (int a = 0; a < PX; a++) {
                    const long long wo = wj + wrap_idx(min(i0 - 2 + bi + a, n1 + 1), n1);
                    u[a] = W[1 * plane + wo];
                    vv[a] = W[2 * plane + wo];
                    w[a] = W[3 * plane + wo];
                    T[a] = W[5 * plane + wo];
                    mu[a] = (R)W[7 * plane + wo];
                }
            } else {
                if (TMA) {
#pragma unroll
                    for (int v = 0; v < 5; v++) ldp<PX>(sq(s, v) + p, q[v]);
                }
#pragma unroll
                for (int a = 0; a < PX; a++) {
                    const double qa[5] = {q[0][a], q[1][a], q[2][a], q[3][a], q[4][a]};
                    prims_from_q(P, qa, u[a], vv[a], w[a], T[a]);
                    mu[a] = mu_of<R>(T[a]);
                }
            }
            stp<PX>((R *)sl.U + p, u);
            stp<PX>((R *)sl.V + p, vv);
            stp<PX>((R *)sl.W + p, w);
            stp<PX>((R *)sl.T + p, T);
            stp<PX>(MU + p, mu);
        };
        // the wall test taken once per plane, so that the loop's body is
        // straight-line code (with per-thread box loads, both of a thread's pairs' are
        // in flight at once; one pair at a time took 2.7% more of the mixed stage time, and
        // loads held across the inviscid sums spill 676 bytes)
        auto loop = [&](bool wall_plane) {
#pragma unroll
            for (int l = 0; l < NL; l++) one(l, wall_plane);
            if (with_xy) inv_xy(m - 1, *Fxy);
        };
        if (wall) loop(true);
        else loop(false);
    };

    // own columns' Q and u,v,w,T of plane m read straight from memory
    auto center = [&](int m, double q[5][PX], double u[PX], double v[PX], double w[PX], double T[PX]) {
        const long long off = (long long)m * plane + colo;
#pragma unroll
        for (int c = 0; c < 5; c++) ldgp<PX>(qin() + c * vol + off, q[c]);
        if (m == 1 || m == n3) {
            const double *W = P.wp + (size_t)(m == 1 ? 0 : 8) * plane + colo;
            ldgp<PX>(W + 1 * plane, u);
            ldgp<PX>(W + 2 * plane, v);
            ldgp<PX>(W + 3 * plane, w);
            ldgp<PX>(W + 5 * plane, T);
        } else {
#pragma unroll
            for (int a = 0; a < PX; a++) {
                const double qa[5] = {q[0][a], q[1][a], q[2][a], q[3][a], q[4][a]};
                prims_from_q(P, qa, u[a], v[a], w[a], T[a]);
            }
        }
    };

    // x and y gradients of a ring field at the own points (and its own values)
    auto grad_x = [&](const R *f, R g[PX], R f0[PX]) {
        if constexpr (PX == 2) {
            R x[6];
            row(f + bc, x);
            g[0] = (x[3] - x[1]) * C.hdx;
            g[1] = (x[4] - x[2]) * C.hdx;
            f0[0] = x[2];
            f0[1] = x[3];
        } else {
            g[0] = (f[bc + 1] - f[bc - 1]) * C.hdx;
            f0[0] = f[bc];
        }
    };
    auto grad_y = [&](const R *f, R g[PX]) {
        R a[PX], b[PX];
        ldp<PX>(f + bc + BX, a);
        ldp<PX>(f + bc - BX, b);
#pragma unroll
        for (int k = 0; k < PX; k++) g[k] = (a[k] - b[k]) * C.hdy;
    };
    auto own = [&](const R *f, R f0[PX]) { ldp<PX>(f + bc, f0); };
    // mu and p = rho T / (gama Ma^2) at the own points: mu at mo, Q slot s, T
    auto mu_p = [&](int mo, int s, const R T0[PX], R mu[PX], R pr[PX]) {
        own(smu(mo), mu);
        own(sq(s, 0), pr);
#pragma unroll
        for (int k = 0; k < PX; k++) pr[k] = (pr[k] * T0[k]) * C.inv_gM2;
    };

    // hD at the own columns of interior plane m (prims at po, mu at mo, Q
    // slot s); dz from (m-1, m+1) values
    auto hflux = [&](int m, int po, int mo, int s, const R um[PX], const R vm[PX], const R wm[PX], const R Tm[PX],
                     const R up[PX], const R vp[PX], const R wp_[PX], const R Tp[PX], R h[PX][4]) {
        const Slot sl = slot(po);
        const R sc = ktab(kCzh, m);
        R ux[PX], vy[PX], wx[PX], wy[PX], u0[PX], v0[PX], w0[PX], T0[PX], mu[PX], pr[PX];
        grad_x(sl.U, ux, u0);
        grad_y(sl.V, vy);
        own(sl.V, v0);
        grad_x(sl.W, wx, w0);
        grad_y(sl.W, wy);
        own(sl.T, T0);
        mu_p(mo, s, T0, mu, pr);
#pragma unroll
        for (int a = 0; a < PX; a++)
            visc_fz_vals(C, ux[a], vy[a], wx[a], wy[a], u0[a], v0[a], w0[a], mu[a], pr[a], (up[a] - um[a]) * sc,
                         (vp[a] - vm[a]) * sc, (wp_[a] - wm[a]) * sc, (Tp[a] - Tm[a]) * sc, h[a]);
    };
    // hD at column `colo + a` of wall plane m, from the wall's own values in
    // memory, in double; one-sided dz against the interior neighbour values
    // (ui..Ti): (q(2)-q(1))/dz1 at the bottom, (q(nP3)-q(nP3-1))/dzN at the
    // top.  The pressure is the pressure-BC state.
    auto hflux_wall = [&](int m, int a, double ui, double vi, double wi, double Ti, double h[4]) {
        const double *W = P.wp + (size_t)(m == 1 ? 0 : 8) * plane + colo + a;
        const long long px = P.px;
        const double u0 = W[plane], v0 = W[2 * plane], w0 = W[3 * plane], T0 = W[5 * plane];
        const double sc = m == 1 ? P.inv_dz1 : P.inv_dzN;
        const double ux = (W[plane + 1] - W[plane - 1]) * P.hdx;
        const double vy = (W[2 * plane + px] - W[2 * plane - px]) * P.hdy;
        const double wx = (W[3 * plane + 1] - W[3 * plane - 1]) * P.hdx;
        const double wy = (W[3 * plane + px] - W[3 * plane - px]) * P.hdy;
        const double uz = (m == 1 ? ui - u0 : u0 - ui) * sc, vz = (m == 1 ? vi - v0 : v0 - vi) * sc;
        const double wz = (m == 1 ? wi - w0 : w0 - wi) * sc, Tz = (m == 1 ? Ti - T0 : T0 - Ti) * sc;
        visc_fz_vals(P.cd, ux, vy, wx, wy, u0, v0, w0, W[7 * plane], W[6 * plane], uz, vz, wz, Tz, h);
    };

    // halo-flux points h: fD of the two x-halo columns at h < 2*TJ, gD of the two
    // y-halo rows from there on.  The x ones are taken by the first warp, the y ones
    // by the next ones, one point per thread (a second one where the CTA has fewer
    // threads).  plane t-1's values (u or v, and w) of point h are kept in sH[.][h].
    auto hbox = [&](int h) -> int {
        if (h < 2 * TJ) {
            const int side = h / TJ, r = h - side * TJ;
            return (r + 2) * BX + (side ? TI + 2 : 1);
        }
        const int side = (h - 2 * TJ) / TI, cc = h - 2 * TJ - side * TI;
        return (side ? TJ + 2 : 1) * BX + cc + 2;
    };
    auto each_halo = [&](auto &&f) {
#pragma unroll
        for (int h0 = 0; h0 < 32 + 2 * TI; h0 += NT) {
            const int l = tid + h0;
            if (l < 2 * TJ) f(l);
            else if (l >= 32 && l < 32 + 2 * TI) f(l - 32 + 2 * TJ);
        }
    };
    // the halo points' values (u or v, w) in ring slot sl, kept as plane t-1
    auto keep_halo = [&](const Slot &sl) {
        each_halo([&](int h) {
            const int b = hbox(h);
            sH[h] = h < 2 * TJ ? sl.U[b] : sl.V[b];
            sH[NHL + h] = sl.W[b];
        });
    };

    // ---------------- prologue: planes kb-1 (Q slot 0, prims at pP) and kb
    // (Q slot 1, prims at pZ); hD(kb-1); plane kb+1 starts its way in
    issue(kb - 1, 0);
    issue(kb, 1);
    issue(kb + 1, 2);   // kb+1 <= ke+1 <= nP3
    issue_base(kb);
    bool bad = !wait_slot(0);
    convert(kb - 1, 0, pP, mP, false);
    bad = !wait_slot(1) || bad;
    convert(kb, 1, pZ, mZ, false);
    if (__syncthreads_or(bad)) { give_up(3); return; }   // slots 0 and 1

    {
        const Slot sA = slot(pP), sB = slot(pZ);
        if (col_ok) {
            R uA[PX], vA[PX], wA[PX], uB[PX], vB[PX], wB[PX], TB[PX];
            own(sA.U, uA); own(sA.V, vA); own(sA.W, wA);
            own(sB.U, uB); own(sB.V, vB); own(sB.W, wB); own(sB.T, TB);
            // hD(kb-1)
            if (kb - 1 == 1) {
#pragma unroll
                for (int a = 0; a < PX; a++) {
                    double h[4];
                    if (a == 0 || i + a <= n1) {
                        hflux_wall(1, a, uB[a], vB[a], wB[a], TB[a], h);
#pragma unroll
                        for (int c = 0; c < 4; c++) h1[a][c] = (R)h[c];
                    }
                }
            } else {
                double q[5][PX], u[PX], v[PX], w[PX], T[PX];
                center(kb - 2, q, u, v, w, T);
                R ur[PX], vr[PX], wr[PX], Tr[PX];
#pragma unroll
                for (int a = 0; a < PX; a++) {
                    ur[a] = (R)u[a]; vr[a] = (R)v[a]; wr[a] = (R)w[a]; Tr[a] = (R)T[a];
                    wm2[a] = wr[a];
#pragma unroll
                    for (int c = 0; c < 5; c++) qm2[c][a] = (R)q[c][a];
                }
                hflux(kb - 1, pP, mP, 0, ur, vr, wr, Tr, uB, vB, wB, TB, h1);
            }
#pragma unroll
            for (int c = 0; c < 5; c++) own(sq(0, c), qm1[c]);
#pragma unroll
            for (int a = 0; a < PX; a++) { um1[a] = uA[a]; vm1[a] = vA[a]; wm1[a] = wA[a]; }
            own(sA.T, Tm1);
        }
        keep_halo(sA);
    }
    __syncthreads();

    // source of plane m: lagged wall-shear forcing (main_v1.9.f90:565-571), formed on
    // every launch (the statistics array always holds these entries) and selected by
    // the flag; buoyancy on the wall-normal momentum and its work on the energy
    auto source = [&](int m, const R u[PX], const R w[PX], const R T[PX], const R r[PX], double s2[PX], double s4[PX],
                      double s5[PX]) {
        const double tau = *stau, rb = rbar(m);
        const double f2 = (0.5 * tau) * rb;
#pragma unroll
        for (int a = 0; a < PX; a++) {
            const double f5 = (((P.ggM * (double)u[a]) * 0.5) * tau) * rb;
            s2[a] = P.force_on ? f2 : 0.0;
            s4[a] = 0.0;
            s5[a] = P.force_on ? f5 : 0.0;
            if (buoy) {
                const double bq = P.ri * ((double)r[a] * ((double)T[a] - P.tref));
                s4[a] = bq;
                s5[a] = s5[a] + (P.ggM * (double)w[a]) * bq;
            }
        }
    };
    // Plane tz completed from what plane tz+2 brings: w and Q of plane tz+2 (wn, getq)
    // and hD(tz+1) (h).  Of the periodic images (the ghosts the reference's halo exchange
    // fills) those in x are stored here, by one predicated store; those in y are whole
    // rows, which the kernel that follows copies (image_body).  With all of them
    // stored here the CTAs at the periodic edges, a third of all, took 10% longer than
    // the others, and the whole launch with them.
    auto complete = [&](int tz, const R wn[PX], const R h[PX][4], bool staged, auto &&getq) {
        const R s12p = ktab(kS12o, tz), czp = ktab(kCzh, tz);
        const long long off = (long long)tz * plane + colo;
        R wq[PX];
        double qu[5][PX];
        [[maybe_unused]] double s2[PX], s4[PX], s5[PX];
#pragma unroll
        for (int a = 0; a < PX; a++) wq[a] = qk[a] ? w4[a] : -(wn[a] * s12p);
        if constexpr (!FOLD) {
            source(tz, um1, wm1, Tm1, qm1[0], s2, s4, s5);
            if (staged) cp_async_wait<0>();
        }
#pragma unroll
        for (int c = 0; c < 5; c++) {
            const int d = c > 0 ? c - 1 : 0;
            R qn[PX];
            getq(c, qn);
            if constexpr (FOLD) {
#pragma unroll
                for (int a = 0; a < PX; a++) {
                    R x = wq[a] * qn[a];
                    if (c > 0) x = fmaR(h[a][d], czp, x);
                    qu[c][a] = qm1[c][a] + fmaR(-(R)P.rk_cdt, x, Fs[a][c]);
                }
            } else {
                // in double, on the stage input at its stored precision
                double qs[PX], qb[PX];
                if (TMA) {
#pragma unroll
                    for (int a = 0; a < PX; a++) qs[a] = (double)qm1[c][a];
                } else if (staged) {
                    ldp<PX>(sQB + (c * NT + tid) * PX, qs);
                } else {
                    ldgp<PX>(qin() + c * vol + off, qs);
                }
                if (need_base) {
                    if (staged) ldp<PX>(sQB + (c * NT + tid) * PX, qb);
                    else ldgp<PX>(P.qbase + c * vol + off, qb);
                }
#pragma unroll
                for (int a = 0; a < PX; a++) {
                    R F = addR(Fs[a][c], fmaR(wq[a], qn[a], H1p[a][c]));
                    if (c > 0) F = fmaR(h[a][d] - hm[a][d], czp, F);
                    double Rd = -(double)F;
                    if (c == 1) Rd = s2[a] - (double)F;
                    if (c == 3 && buoy) Rd = s4[a] - (double)F;
                    if (c == 4) Rd = s5[a] - (double)F;
                    if (need_base) qu[c][a] = (P.rk_a * qb[a] + P.rk_b * qs[a]) + P.rk_cdt * Rd;
                    else qu[c][a] = qs[a] + P.rk_cdt * Rd;
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 5; c++) {
            QO *O = qout() + c * vol + off;
            if (PX == 1 || out1) stp<PX>(O, qu[c]);
            else *O = (QO)qu[c][0];
        }
        if (xim != 0) {
#pragma unroll
            for (int a = 0; a < PX; a++) {
                const int ia = i + a;
                if (PX > 1 && !(ia <= 3 || (ia >= n1 - 2 && ia <= n1 - 1))) continue;
                QO *O = qout() + off + a + xim;
#pragma unroll
                for (int c = 0; c < 5; c++) O[c * vol] = (QO)qu[c][a];
            }
        }
        // the blow-up test: rho, rho*rhoE - ggM/2 |rho u|^2 (the sign of T), all finite
        if constexpr (CHK) {
            if (P.check) {
#pragma unroll
                for (int a = 0; a < PX; a++) {
                    if (a == 1 && !out1) break;
                    const double tr = qu[0][a] * qu[4][a] -
                                      P.ggMh * ((qu[1][a] * qu[1][a] + qu[2][a] * qu[2][a]) + qu[3][a] * qu[3][a]);
                    if (qu[0][a] < 0.0 || (qu[0][a] > 0.0 && tr < 0.0)) flag_blown(P.status, i + a, j, tz, kstep(P));
                    bool fin = true;
#pragma unroll
                    for (int c = 0; c < 5; c++) fin = fin && isfinite(qu[c][a]);
                    if (!fin) flag_nonfinite(P.status, i + a, j, tz);
                }
            }
        }
    };
    // float rings: the own points' RK base of plane m starts its way into shared memory;
    // in the stage that reads the double state, which has no other base, that state (read
    // from memory by the update it took 2.3% more of the mixed stage time)
    auto fetch_base = [&](int m) {
        if (!FOLD && out0) {
            const double *src = (TMA ? P.qbase : reinterpret_cast<const double *>(qin())) + (long long)m * plane + colo;
#pragma unroll
            for (int c = 0; c < 5; c++) cp_async_d<PX>(sQB + (c * NT + tid) * PX, src + c * vol);
        }
        if (!FOLD) cp_async_commit();
    };

    // Iteration t forms the fluxes of plane t and completes plane t-1, whose
    // wall-normal derivatives need hD(t) and Q, w of plane t+1.  So plane t+1 is
    // the furthest plane read, each point is converted once, hD shares the
    // gradients of fD and gD, and no own column is read from memory on the way.
    // Plane ke is completed after the loop, from its own columns alone.
    for (int t = kb; t <= ke; t++) {
        // ---------- A: plane t+1's box is converted, beside the inviscid x/y sums of
        // plane t; after the barrier, plane t+2's box starts its way in (converted
        // at the next plane).
        // No barrier ends the plane, so a warp that has finished plane t goes on to
        // plane t+1's box wait and conversion while others still run phase E.  What
        // makes that safe: plane t+2's box goes into the slot of plane t-1, and plane
        // t-1's RK base over plane t-2's, only after
        // phase A's barrier, which every thread passes after its phase-E reads of that
        // slot; and phase E reads no primitive or mu slot, which the next conversion
        // overwrites.
        R Fxy[PX][5];
        if (t > kb) fetch_base(t - 1);
        bad = !wait_slot(iP) || bad;
        if (FOLD && need_base) bad = !wait_slot(3) || bad;
        convert(t + 1, iP, pP, mP, true, &Fxy);
        if (__syncthreads_or(bad)) { give_up(15); return; }   // every slot in use
        if (t < ke) {
            issue(t + 2, iN);
            issue_base(t + 1);
        }

        // ---------- C: viscous flux vectors
        const R czt = ktab(kCzh, t);
        const Slot s0 = slot(pZ), sp = slot(pP);
        R h[PX][4], wn[PX], w0[PX], u0[PX], v0[PX], T0[PX];
        if (col_ok) {
            R ux[PX], uy[PX], vx[PX], vy[PX], wx[PX], wy[PX], Tx[PX], Ty[PX], pr[PX], un[PX], vn[PX], Tn[PX], mu[PX], m3[PX];
            own(sp.U, un); own(sp.V, vn); own(sp.W, wn); own(sp.T, Tn);
            grad_x(s0.U, ux, u0); grad_y(s0.U, uy);
            grad_x(s0.V, vx, v0); grad_y(s0.V, vy);
            grad_x(s0.W, wx, w0); grad_y(s0.W, wy);
            grad_x(s0.T, Tx, T0); grad_y(s0.T, Ty);
            mu_p(mZ, iZ, T0, mu, pr);
            if constexpr (!FOLD) {
                own(sq(iZ, 3), m3);
                const R pez = ktab(kPez, t);
#pragma unroll
                for (int a = 0; a < PX; a++) qz[a] = (pez * fabs(m3[a])) > C.pez_val * mu[a];
            }
            R f[PX][4], g[PX][4];
#pragma unroll
            for (int a = 0; a < PX; a++) {
                const R uz = (un[a] - um1[a]) * czt, vz = (vn[a] - vm1[a]) * czt, wz = (wn[a] - wm1[a]) * czt;
                const R Tz = (Tn[a] - Tm1[a]) * czt;
                fd_point(C, mu[a], pr[a], u0[a], v0[a], w0[a], ux[a], vy[a], wz, vx[a], uy[a], wx[a], uz, Tx[a], f[a]);
                gd_point(C, mu[a], pr[a], u0[a], v0[a], w0[a], ux[a], vy[a], wz, vx[a], uy[a], wy[a], vz, Ty[a], g[a]);
                visc_fz_vals(C, ux[a], vy[a], wx[a], wy[a], u0[a], v0[a], w0[a], mu[a], pr[a], uz, vz, wz, Tz, h[a]);
            }
#pragma unroll
            for (int c = 0; c < 4; c++) {
                R x[PX], y[PX];
#pragma unroll
                for (int a = 0; a < PX; a++) { x[a] = f[a][c]; y[a] = g[a][c]; }
                // fD3 and gD2 are one stress
                if (c == 1) stp<PX>(sX + (ty + 1) * FP + PX * tx + FO, x);
                else stp<PX>(sF + ((c > 1 ? c - 1 : c) * TJ + ty) * FP + PX * tx + FO, x);
                if (c > 0) stp<PX>(sG + ((c - 1) * (TJ + 2) + ty + 1) * TI + PX * tx, y);
            }
        }
        {
            const R *MU = smu(mZ), *RHO = sq(iZ, 0);
            each_halo([&](int hp) {
                if (hp < 2 * TJ) {
                    const int side = hp / TJ, r = hp - side * TJ;
                    const int ci = side ? i0 + TI : i0 - 1, cj = j0 + r;
                    if (ci <= n1 && cj <= n2) {
                        R f[4];
                        visc_fx<BX, R>(C, s0, sH[hp], sH[NHL + hp], sp, MU, RHO, hbox(hp), czt, f);
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            const int o = side ? FO + TI : FO - 1;
                            if (c == 1) sX[(r + 1) * FP + o] = f[c];
                            else sF[((c > 1 ? c - 1 : c) * TJ + r) * FP + o] = f[c];
                        }
                    }
                } else {
                    const int side = (hp - 2 * TJ) / TI, cc = hp - 2 * TJ - side * TI;
                    const int ci = i0 + cc, cj = side ? j0 + TJ : j0 - 1;
                    if (ci <= n1 && cj <= n2) {
                        R g[4];
                        visc_fy<BX, R>(C, s0, sH[hp], sH[NHL + hp], sp, MU, RHO, hbox(hp), czt, g);
#pragma unroll
                        for (int c = 1; c < 4; c++) sG[(c - 1) * S::NGY + (side ? TJ + 1 : 0) * TI + cc] = g[c];
                        sX[(side ? TJ + 1 : 0) * FP + FO + cc] = g[0];
                    }
                }
            });
            keep_halo(s0);
        }
        __syncthreads();
        // ---------- E: (FP64: plane t-1 completed;) the flux derivatives of plane t known
        // so far.  In FP64 the three loops below stay apart: merged, their live values
        // spill, and with two CTAs' shared memory the L1 has no room for spills.
        if (t > kb && out0) complete(t - 1, wn, h, true, [&](int c, R qn[PX]) { own(sq(iP, c), qn); });
        if (col_ok) {
#pragma unroll
            for (int a = 0; a < PX; a++) { um1[a] = u0[a]; vm1[a] = v0[a]; Tm1[a] = T0[a]; }
        }
        if (out0) {
            const R s12 = ktab(kS12, t), s12o = ktab(kS12o, t), s8 = ktab(kS8, t);
            R w[PX][5];
#pragma unroll
            for (int a = 0; a < PX; a++) {
                qk[a] = qz[a];
                inv_weights(wm2[a], wm1[a], w0[a], wn[a], R(0), qk[a], s8, s12, s12o, w[a]);
                w4[a] = w[a][4];   // of the QUICK set; the central one needs w(t+2)
                wm2[a] = wm1[a];
                wm1[a] = w0[a];
            }
            double s2[PX], s4[PX], s5[PX];
            if constexpr (FOLD) {
                R r0[PX];
                own(sq(iZ, 0), r0);
                source(t, um1, w0, Tm1, r0, s2, s4, s5);
            }
#pragma unroll
            for (int c = 0; c < 5; c++) {
                const int d = c > 0 ? c - 1 : 0;
                R qn[PX], q0[PX];
                own(sq(iP, c), qn);
                own(sq(iZ, c), q0);
#pragma unroll
                for (int a = 0; a < PX; a++) {
                    R H;
                    if constexpr (FOLD) {
                        H = fmaR(w[a][3], qn[a], fmaR(w[a][2], q0[a], w[a][1] * qm1[c][a]));
                        if (c == 1) H = H - s2[a];
                        if (c == 3 && buoy) H = H - s4[a];
                        if (c == 4) H = H - s5[a];
                        Fs[a][c] = fmaR(-P.rk_cdt, H, Fxy[a][c]);
                    } else {
                        H1p[a][c] = H = wsum4(w[a], qm2[c][a], qm1[c][a], q0[a], qn[a]);
                        Fs[a][c] = Fxy[a][c];
                        if (c > 0) hm[a][d] = h1[a][d];
                    }
                    if (c > 0) h1[a][d] = h[a][d];
                    qm2[c][a] = qm1[c][a];
                    qm1[c][a] = q0[a];
                }
            }
#pragma unroll
            for (int c = 1; c < 5; c++) {
                // fD2, fD3, fD4, fD5 and gD2, gD3, gD4, gD5
                const R *F = (c == 2 ? sX + (ty + 1) * FP : sF + ((c > 2 ? c - 2 : c - 1) * TJ + ty) * FP) + PX * tx + FO;
                const R *G = c == 1 ? sX + ty * FP + PX * tx + FO : sG + ((c - 2) * (TJ + 2) + ty) * TI + PX * tx;
                const int gs = 2 * (c == 1 ? FP : TI);
                R F2[PX], gm[PX], gp[PX];
                if constexpr (PX == 2) {
                    R x[6];
                    row(F, x);
                    F2[0] = x[3] - x[1];
                    F2[1] = x[4] - x[2];
                } else {
                    F2[0] = F[1] - F[-1];
                }
                ldp<PX>(G, gm);
                ldp<PX>(G + gs, gp);
#pragma unroll
                for (int a = 0; a < PX; a++) {
                    if constexpr (FOLD)
                        Fs[a][c] = fmaR(-P.rk_cdt, fmaR(gp[a] - gm[a], C.hdy, F2[a] * C.hdx), Fs[a][c]);
                    else
                        Fs[a][c] = fmaR(gp[a] - gm[a], C.hdy, fmaR(F2[a], C.hdx, Fs[a][c]));
                }
            }
        } else if (col_ok) {
            // a column whose fD or gD a neighbour reads
#pragma unroll
            for (int a = 0; a < PX; a++) wm1[a] = w0[a];
        }
        {
            const int o = iZ;
            iZ = iP; iP = iN; iN = o;
            int x = pZ; pZ = pP; pP = x;
            x = mZ; mZ = mP; mP = x;
        }
    }
    if (!out0) return;
    // ---------- plane ke completed: hD(ke+1) from the converted plane ke+1 and plane
    // ke+2 in memory, or the top wall's (its own values in memory, against plane
    // nP3-1's)
    R h[PX][4], qn[5][PX], wn[PX] = {};
    double q[5][PX], u[PX], v[PX], w[PX], T[PX];
    if (ke + 1 == n3) {
        center(n3 - 1, q, u, v, w, T);
#pragma unroll
        for (int a = 0; a < PX; a++) {
            double hw[4];
            hflux_wall(n3, a, u[a], v[a], w[a], T[a], hw);
#pragma unroll
            for (int c = 0; c < 4; c++) h[a][c] = (R)hw[c];
#pragma unroll
            for (int c = 0; c < 5; c++) qn[c][a] = R(0);
        }
    } else {
        center(ke + 2, q, u, v, w, T);
        R un[PX], vn[PX], Tn[PX];
#pragma unroll
        for (int a = 0; a < PX; a++) {
            un[a] = (R)u[a]; vn[a] = (R)v[a]; wn[a] = (R)w[a]; Tn[a] = (R)T[a];
#pragma unroll
            for (int c = 0; c < 5; c++) qn[c][a] = (R)q[c][a];
        }
        hflux(ke + 1, pZ, mZ, iZ, um1, vm1, wm1, Tm1, un, vn, wn, Tn, h);
    }
    complete(ke, wn, h, false, [&](int c, R x[PX]) {
#pragma unroll
        for (int a = 0; a < PX; a++) x[a] = qn[c][a];
    });
}

template <int TI, int TJ, typename QI, typename QO, typename R, bool BUOY>
__global__ void __launch_bounds__(StageShape<TI, TJ, R>::NT, StageShape<TI, TJ, R>::minb)
    k_stage(const KParams P, const __grid_constant__ CUtensorMap tmq, const __grid_constant__ CUtensorMap tmb)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    grid_dep_enter();
    stage_body<TI, TJ, QI, QO, R, BUOY ? 1 : 0, false>(P, &tmq, &tmb, blockIdx.x, blockIdx.y, blockIdx.z, threadIdx.x,
                                                       threadIdx.y, smem_raw, nullptr);
}

// ---------------------------------------------------------------------------
// Wall BC + pressure BC (main_v1.9.f90:623-720 on the two wall planes).
// One thread per (i,j) of a wall plane, ghosts included.

// point p of an n1 x n2 x .. box (i fastest), 0-based.  32-bit unsigned: device memory holds
// fewer than 2^31 points, and the 64-bit quotients it replaces cost more than the loads
__device__ __forceinline__ void split3(unsigned p, unsigned n1, unsigned n2, int &i, int &j, int &k)
{
    const unsigned r = p / n1, l = r / n2;
    i = (int)(p - r * n1);
    j = (int)(r - l * n2);
    k = (int)l;
}

// var(u, v, T) of an interior point as the reference holds it (corner columns
// keep their stale values)
template <typename QT>
__device__ __forceinline__ void inner_uvT(const KParams &P, int i, int j, int k, double &u, double &v, double &T)
{
    const QT *qo = static_cast<const QT *>(P.qout);
    const int n1 = P.n1, n2 = P.n2;
    if ((i == 1 || i == n1) && (j == 1 || j == n2)) {
        const double *C = P.cs + ((size_t)k * 4 + (i == 1 ? 0 : 1) + (j == 1 ? 0 : 2)) * 7;
        u = C[1]; v = C[2]; T = C[5];
        return;
    }
    // a periodic duplicate row: its source (the row itself is being written by image blocks)
    const long long o = (long long)k * P.plane + (long long)wrap_idx(j, n2) * P.px + i;
    const double q0 = qo[o];
#ifndef CHAN_TRUE_DIV
    const double r = rcp_fast(q0);
    u = (double)qo[P.vol + o] * r;
    v = (double)qo[2 * P.vol + o] * r;
    const double w = (double)qo[3 * P.vol + o] * r;
    const double E = (double)qo[4 * P.vol + o] * r;
#else
    u = (double)qo[P.vol + o] / q0;
    v = (double)qo[2 * P.vol + o] / q0;
    const double w = (double)qo[3 * P.vol + o] / q0;
    const double E = (double)qo[4 * P.vol + o] / q0;
#endif
    T = E - P.ggMh * ((u * u + v * v) + w * w);
}

// wall values u, v, T of point (i,j) of wall `wall` after the wall BC
template <typename QT>
__device__ void wall_point(const KParams &P, int wall, int i, int j, double &u, double &v, double &T)
{
    const WallBC &B = P.wbc[wall];
    const int n1 = P.n1, n2 = P.n2;
    const int ic = i < 1 ? 1 : (i > n1 ? n1 : i), jc = j < 1 ? 1 : (j > n2 ? n2 : j);
    const int k2 = wall == 0 ? 2 : P.n3 - 1, k3 = wall == 0 ? 3 : P.n3 - 2;
    const double *c = wall == 0 ? P.f1 : P.b1;
    u = 0.0;
    v = 0.0;
    double u2 = 0, v2 = 0, T2 = 0, u3 = 0, v3 = 0, T3 = 0;
    const bool need_inner = (B.vel == 1 && B.mask[(jc - 1) * n1 + ic - 1]) || B.therm == 1;
    if (need_inner) {
        inner_uvT<QT>(P, ic, jc, k2, u2, v2, T2);
        inner_uvT<QT>(P, ic, jc, k3, u3, v3, T3);
    }
    if (B.vel == 1) {
        if (B.mask[(jc - 1) * n1 + ic - 1]) {
            u = ((B.g - c[1] * u2) - c[2] * u3) / c[0];
            v = ((B.g - c[1] * v2) - c[2] * v3) / c[0];
        }
    } else if (B.vel == 2) {
        u = B.uv[(jc - 1) * n1 + ic - 1];
        v = B.uv[n1 * n2 + (jc - 1) * n1 + ic - 1];
    } else if (B.vel == 3) {
        const double x = B.x1[ic - 1];
        v = B.A * sin((B.kx * x + B.om * ktime(P)) + ((jc & 1) ? B.ph : 0.0));
    }
    T = (B.therm == 1) ? ((B.dTdz - c[1] * T2) - c[2] * T3) / c[0] : B.Tw;
}

// QT: storage type of the stage output the wall BC reads (the planes next to the wall)
constexpr int kWallBX = 32, kWallBY = 8;
constexpr int kWallHX = kWallBX + 2, kWallHY = kWallBY + 2;
using WallStage = double[2][6][kWallHY][kWallHX];

// One block's work of the wall kernel: block (bx, by) of wall `wall`, by NTH
// threads, near-wall staging area sp.
template <typename QT, int NTH>
__device__ __forceinline__ void wall_body(const KParams &P, int bx_, int by_, int wall, int tid, WallStage &sp)
{
    const QT *qo = static_cast<const QT *>(P.qout);
    const int n1 = P.n1, n2 = P.n2, n3 = P.n3;
    const long long plane = P.plane, vol = P.vol;
    // primitives of the two planes next to the wall on the block's (i,j) tile
    // plus a 1-point halo, each computed once: [plane][r,u,v,w,p,mu][by][bx]
    constexpr int HX = kWallHX, HY = kWallHY;
    {
        const int k2 = wall == 0 ? 2 : n3 - 1, k3 = wall == 0 ? 3 : n3 - 2;
        const int i0 = bx_ * kWallBX - 1, j0 = by_ * kWallBY - 1;
        for (int e = tid; e < 2 * HX * HY; e += NTH) {
            const int pl = e / (HX * HY), r0 = e - pl * HX * HY, by = r0 / HX, bx = r0 - by * HX;
            const int ii = i0 + bx, jj = j0 + by;
            if (ii < 1 || ii > n1 || jj < 1 || jj > n2) continue;
            // a periodic duplicate row: its source (the row itself is being written by
            // the image blocks)
            const long long o = (long long)(pl == 0 ? k2 : k3) * plane + (long long)wrap_idx(jj, n2) * P.px + ii;
            const double q0 = qo[o], q1 = qo[vol + o], q2 = qo[2 * vol + o];
            const double q3 = qo[3 * vol + o], q4 = qo[4 * vol + o];
#ifndef CHAN_TRUE_DIV
            const double r = rcp_fast(q0);
            const double u = q1 * r, v = q2 * r, w = q3 * r;
            const double E = q4 * r;
#else
            const double u = q1 / q0, v = q2 / q0, w = q3 / q0;
            const double E = q4 / q0;
#endif
            const double T = E - P.ggMh * ((u * u + v * v) + w * w);
            sp[pl][0][by][bx] = q0;
            sp[pl][1][by][bx] = u;
            sp[pl][2][by][bx] = v;
            sp[pl][3][by][bx] = w;
#ifndef CHAN_TRUE_DIV
            sp[pl][4][by][bx] = (q0 * T) * P.inv_gM2;
#else
            sp[pl][4][by][bx] = (q0 * T) / P.gM2;
#endif
            sp[pl][5][by][bx] = pow07(T);
        }
    }
    __syncthreads();
    if (frozen(P.status, kstep(P))) return;
    double *W = P.wp + (size_t)wall * 8 * plane;
#pragma unroll 1
    for (int e = tid; e < kWallBX * kWallBY; e += NTH) {
        const int i = bx_ * kWallBX + e % kWallBX;
        const int j = by_ * kWallBY + e / kWallBX;
        if (i > n1 + 1 || j > n2 + 1) continue;
        const long long idx = (long long)j * P.px + i;
        const bool custom = P.wall_custom != 0;
        double uw = 0.0, vw = 0.0, Tw = wall == 0 ? P.Twb : P.Twt;
        double muw = wall == 0 ? P.muwb : P.muwt;
        if (custom) {
            wall_point<QT>(P, wall, i, j, uw, vw, Tw);
            if (P.wbc[wall].therm == 1) muw = pow07(Tw);
        }
        const double pold = W[6 * plane + idx];
        const double rho = (P.gM2 * pold) / Tw;   // gama*Mac**2*p/T with the previous p
        double pnew = pold;
        if (i >= 2 && i <= n1 - 1 && j >= 2 && j <= n2 - 1) {
            // neighbours at the two planes next to the wall: k2 (adjacent) and k3
            const int k2 = wall == 0 ? 2 : n3 - 1, k3 = wall == 0 ? 3 : n3 - 2;
            const double *c1 = wall == 0 ? P.f1 : P.b1;
            const double *c2 = wall == 0 ? P.f2 : P.b2;
            // primitive + mu of one interior point, as calcPrim/calcBC produce them
            // (staged above); kk selects the plane k2 or k3
            auto prim = [&](int ii, int jj, int kk, double &r, double &u, double &v, double &w, double &T,
                            double &p, double &mu) {
                const int pl = kk == k2 ? 0 : 1;
                const int bx = ii - bx_ * kWallBX + 1, by = jj - by_ * kWallBY + 1;
                r = sp[pl][0][by][bx];
                u = sp[pl][1][by][bx];
                v = sp[pl][2][by][bx];
                w = sp[pl][3][by][bx];
                p = sp[pl][4][by][bx];
                mu = sp[pl][5][by][bx];
                T = 0.0;
            };
            // wall-point terms c0*mu_w*u_w of the neighbours (zero for a no-slip wall)
            double t_ip = 0.0, t_im = 0.0, t_jp = 0.0, t_jm = 0.0;
            if (custom) {
                double u, v, T;
                wall_point<QT>(P, wall, i + 1, j, u, v, T);
                t_ip = c1[0] * (P.wbc[wall].therm == 1 ? pow07(T) : muw) * u;
                wall_point<QT>(P, wall, i - 1, j, u, v, T);
                t_im = c1[0] * (P.wbc[wall].therm == 1 ? pow07(T) : muw) * u;
                wall_point<QT>(P, wall, i, j + 1, u, v, T);
                t_jp = c1[0] * (P.wbc[wall].therm == 1 ? pow07(T) : muw) * v;
                wall_point<QT>(P, wall, i, j - 1, u, v, T);
                t_jm = c1[0] * (P.wbc[wall].therm == 1 ? pow07(T) : muw) * v;
            }
            double r, u, v, w, T, p, mu;
            double a2, a3, b2, b3;
            // d/dx of mu*du/dz
            prim(i + 1, j, k2, r, u, v, w, T, p, mu); a2 = c1[1] * mu * u;
            prim(i + 1, j, k3, r, u, v, w, T, p, mu); a3 = c1[2] * mu * u;
            prim(i - 1, j, k2, r, u, v, w, T, p, mu); b2 = c1[1] * mu * u;
            prim(i - 1, j, k3, r, u, v, w, T, p, mu); b3 = c1[2] * mu * u;
            const double dudxdz = (((t_ip + a2) + a3) - ((t_im + b2) + b3)) * P.hdx;
            prim(i, j + 1, k2, r, u, v, w, T, p, mu); a2 = c1[1] * mu * v;
            prim(i, j + 1, k3, r, u, v, w, T, p, mu); a3 = c1[2] * mu * v;
            prim(i, j - 1, k2, r, u, v, w, T, p, mu); b2 = c1[1] * mu * v;
            prim(i, j - 1, k3, r, u, v, w, T, p, mu); b3 = c1[2] * mu * v;
            const double dvdydz = (((t_jp + a2) + a3) - ((t_jm + b2) + b3)) * P.hdy;
            double p2, p3, d2, d3, e2, e3;
            prim(i, j, k2, r, u, v, w, T, p, mu);
            d2 = c2[1] * mu * w; e2 = c1[1] * r * (w * w); p2 = p;
            prim(i, j, k3, r, u, v, w, T, p, mu);
            d3 = c2[2] * mu * w; e3 = c1[2] * r * (w * w); p3 = p;
            // the wall-point w terms vanish: w = 0 on every wall
            const double d2wdz2 = d2 + d3;
            const double drhow2dz = e2 + e3;
            const double lhs = P.invRe * ((-dudxdz - dvdydz) + P.two3rd * ((dudxdz + dvdydz) - 2.0 * d2wdz2)) + drhow2dz;
            pnew = -((lhs + c1[1] * p2) + c1[2] * p3) / c1[0];
        }
        W[0 * plane + idx] = rho;
        W[1 * plane + idx] = uw;
        W[2 * plane + idx] = vw;
        W[3 * plane + idx] = 0.0;
        W[4 * plane + idx] = custom ? Tw + P.ggMh * ((uw * uw + vw * vw) + 0.0) : Tw;
        W[5 * plane + idx] = Tw;
        W[6 * plane + idx] = pnew;
        W[7 * plane + idx] = muw;
        if (P.check && i >= 1 && i <= n1 && j >= 1 && j <= n2) {
            if (rho < 0.0 || Tw < 0.0) flag_blown(P.status, i, j, wall == 0 ? 1 : n3, kstep(P));
            if (!isfinite(rho) || !isfinite(pnew)) flag_nonfinite(P.status, i, j, wall == 0 ? 1 : n3);
        }
    }
}

// Periodic images of the stage output in y: the ghost rows 0, 1, nP2, nP2+1 of
// interior plane k, whole rows (their x images came with the stage), by one block of
// NTH threads; b < image_blocks splits the row points.  The five variables of a point
// at once, so that their loads are in flight together.
constexpr int kImgItems = 512;
__host__ __device__ __forceinline__ int image_blocks(int n1) { return (4 * (n1 + 2) + kImgItems - 1) / kImgItems; }
template <typename QT, int NTH>
__device__ __forceinline__ void image_body(const KParams &P, int k, int b, int tid)
{
    if (frozen(P.status, kstep(P))) return;
    const int n1 = P.n1, n2 = P.n2, px = P.px, n = 4 * (n1 + 2);
    QT *q = static_cast<QT *>(P.qout) + (long long)k * P.plane;
#pragma unroll 2
    for (int e = b * kImgItems + tid; e < min(n, (b + 1) * kImgItems); e += NTH) {
        const int g = e / (n1 + 2), i = e - g * (n1 + 2);
        const int j = g < 2 ? g : n2 + g - 2;
        const QT *r = q + (long long)wrap_idx(j, n2) * px + i;
        QT *o = q + (long long)j * px + i;
        QT x[5];
#pragma unroll
        for (int c = 0; c < 5; c++) x[c] = r[c * P.vol];
#pragma unroll
        for (int c = 0; c < 5; c++) o[c * P.vol] = x[c];
    }
}

// Blocks of the launch that follows a stage: first the wall blocks (x, y, wall), then
// the image blocks of each interior plane.
__host__ __device__ __forceinline__ int wall_blocks_x(int n1) { return (n1 + 2 + kWallBX - 1) / kWallBX; }
__host__ __device__ __forceinline__ int wall_blocks_y(int n2) { return (n2 + 2 + kWallBY - 1) / kWallBY; }
__host__ __device__ __forceinline__ int edge_blocks(int n1, int n2, int n3)
{
    return 2 * wall_blocks_x(n1) * wall_blocks_y(n2) + image_blocks(n1) * (n3 - 2);
}
template <typename QT, int NTH>
__device__ __forceinline__ void edge_body(const KParams &P, int b, int tid, WallStage &sp)
{
    const int nx = wall_blocks_x(P.n1), ny = wall_blocks_y(P.n2), nw = 2 * nx * ny;
    if (b < nw) {
        const int bx = b % nx, r = b / nx;
        wall_body<QT, NTH>(P, bx, r % ny, r / ny, tid, sp);
    } else {
        const int ni = image_blocks(P.n1);
        image_body<QT, NTH>(P, 2 + (b - nw) / ni, (b - nw) % ni, tid);
    }
}

template <typename QT>
__global__ void __launch_bounds__(kWallBX * kWallBY, 4) k_wall(const KParams P)
{
    __shared__ double sp[2][6][kWallHY][kWallHX];
    grid_dep_enter();
    edge_body<QT, kWallBX * kWallBY>(P, blockIdx.x, threadIdx.x, sp);
}

// ---------------------------------------------------------------------------
// var(i,j,k,1:7) as the reference holds it after a stage (used by the
// statistics, the blow-up scan and downloads).
__device__ __forceinline__ void ref_var(const KParams &P, const double *q, int i, int j, int k, double x[7])
{
    const int n1 = P.n1, n2 = P.n2, n3 = P.n3;
    if (k == 1 || k == n3) {
        const double *W = P.wp + (size_t)(k == 1 ? 0 : 8) * P.plane + (long long)j * P.px + i;
        x[0] = W[0]; x[1] = W[P.plane]; x[2] = W[2 * P.plane]; x[3] = W[3 * P.plane];
        x[4] = W[4 * P.plane]; x[5] = W[5 * P.plane]; x[6] = W[6 * P.plane];
        return;
    }
    const bool ci = (i == 1 || i == n1), cj = (j == 1 || j == n2);
    if (ci && cj) {
        const int c = (i == 1 ? 0 : 1) + (j == 1 ? 0 : 2);
        const double *C = P.cs + ((size_t)k * 4 + c) * 7;
#pragma unroll
        for (int m = 0; m < 7; m++) x[m] = C[m];
        return;
    }
    const long long o = (long long)k * P.plane + (long long)j * P.px + i;
    const double q0 = q[o];
    x[0] = q0;
#ifndef CHAN_TRUE_DIV
    // one reciprocal for the four quotients (within an ulp or two of them; the
    // four true divisions, CHAN_TRUE_DIV, cost 0.65% of the step in this and the
    // wall kernel)
    const double r = rcp_fast(q0);
    x[1] = q[P.vol + o] * r;
    x[2] = q[2 * P.vol + o] * r;
    x[3] = q[3 * P.vol + o] * r;
    x[4] = q[4 * P.vol + o] * r;
    x[5] = x[4] - P.ggMh * ((x[1] * x[1] + x[2] * x[2]) + x[3] * x[3]);
    x[6] = (x[0] * x[5]) * P.inv_gM2;
#else
    x[1] = q[P.vol + o] / q0;
    x[2] = q[2 * P.vol + o] / q0;
    x[3] = q[3 * P.vol + o] / q0;
    x[4] = q[4 * P.vol + o] / q0;
    x[5] = x[4] - P.ggMh * ((x[1] * x[1] + x[2] * x[2]) + x[3] * x[3]);
    x[6] = (x[0] * x[5]) / P.gM2;
#endif
}

// Plane moments (avgSpatial, main_v1.9.f90:995-1025) and wall shear
// (calcTauWall, main_v1.9.f90:930-977), in two passes.
constexpr int kStatThreads = 256;

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Pass 1: block (pb, sub) sums the points sub, sub+S, ... (in units of
// kStatThreads) of plane pb (pb < n3: the 23 moment sums of plane k = pb+1;
// pb = n3, n3+1: the wall-shear sum of the bottom, top wall) into
// part[(pb*S + sub)*23 + c].  Pass 2 adds the S partial sums in a fixed
// order: the result is deterministic.
// NTH < kStatThreads threads take the points of kStatThreads in turn, each
// group of 32 with the same points and the same sums.
using StatRed = double[kStatThreads / 32][23];
template <int NTH>
__device__ __forceinline__ void stats_part_body(const KParams &P, const double *q, int do_moments, int do_tau, int S,
                                                double *part, int blk, int tid, StatRed &red)
{
    const int n1 = P.n1, n2 = P.n2, n3 = P.n3;
    const int pb = blk / S, sub = blk - pb * S;
    const int lane = tid & 31;
    if (frozen(P.status, kstep(P) + 1)) return;
    double *out = part + ((size_t)pb * S + sub) * 23;
    if (pb < n3) {
        if (!do_moments) return;
        const int k = pb + 1;
#pragma unroll 1
        for (int v = tid; v < kStatThreads; v += NTH) {
        double acc[23];
#pragma unroll
        for (int c = 0; c < 23; c++) acc[c] = 0.0;
        const int np = n1 * n2;
#pragma unroll 2
        for (int p = sub * kStatThreads + v; p < np; p += S * kStatThreads) {
            const int jj = p / n1, ii = p - jj * n1;
            double x[7];
            ref_var(P, q, ii + 1, jj + 1, k, x);
#pragma unroll
            for (int m = 0; m < 7; m++) {
                acc[m] += x[m];
                acc[7 + m] += x[m] * x[m];
            }
            acc[14] += x[0] * x[3];
            acc[15] += x[0] * x[5];
            acc[16] += x[1] * x[2];
            acc[17] += x[1] * x[3];
            acc[18] += x[2] * x[3];
            acc[19] += x[2] * x[5];
            acc[20] += x[5] * x[3];
            acc[21] += x[6] * x[3];
            acc[22] += x[6] * x[5];
        }
#pragma unroll
        for (int c = 0; c < 23; c++) {
            const double s = warp_sum(acc[c]);
            if (lane == 0) red[v >> 5][c] = s;
        }
        }
        __syncthreads();
        if (tid < 23) {
            double s = 0.0;
            for (int w = 0; w < kStatThreads / 32; w++) s += red[w][tid];
            out[tid] = s;
        }
        return;
    }
    if (!do_tau) return;
    const int wall = pb - n3;
    const double *W = P.wp + (size_t)wall * 8 * P.plane;
    const double *c = wall == 0 ? P.f1 : P.b1;
    const int k2 = wall == 0 ? 2 : n3 - 1, k3 = wall == 0 ? 3 : n3 - 2;
    const int ni = n1 - 2, np = (n1 - 2) * (n2 - 2);
#pragma unroll 1
    for (int v = tid; v < kStatThreads; v += NTH) {
    double acc = 0.0;
    for (int p = sub * kStatThreads + v; p < np; p += S * kStatThreads) {
        const int jj = 2 + p / ni, ii = 2 + p % ni;
        const long long o = (long long)jj * P.px + ii;
        const double mu = W[7 * P.plane + o];
        const double dwdx = ((mu * (W[3 * P.plane + o + 1] - W[3 * P.plane + o - 1])) * 0.5) * P.invdx;
        const long long o2 = (long long)k2 * P.plane + o, o3 = (long long)k3 * P.plane + o;
        const double u2 = q[P.vol + o2] / q[o2];
        const double u3 = q[P.vol + o3] / q[o3];
        const double dudz = mu * ((c[0] * W[1 * P.plane + o] + c[1] * u2) + c[2] * u3);
        acc += (dwdx + dudz) * P.invRe;
    }
    const double s = warp_sum(acc);
    if (lane == 0) red[v >> 5][0] = s;
    }
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < kStatThreads / 32; w++) t += red[w][0];
        out[0] = t;
    }
}

__global__ void __launch_bounds__(kStatThreads, 3) k_stats_part(const KParams P, const double *q, int do_moments,
                                                             int do_tau, int S, double *part)
{
    __shared__ double red[kStatThreads / 32][23];
    grid_dep_enter();
    stats_part_body<kStatThreads>(P, q, do_moments, do_tau, S, part, blockIdx.x, threadIdx.x, red);
}

// Pass 2: one warp per plane / wall adds the S partial sums in order and
// writes stat1Spc, stat2Spc, corrSpc (divided by nP1*nP2) and tauL, tauU
// (divided by (nP1-2)*(nP2-2)); with time averaging on, also adds them into tacc.
__device__ __forceinline__ void stats_fin_body(const KParams &P, int do_moments, int do_tau, int S, const double *part,
                                               int pb, int c)
{
    const int n1 = P.n1, n2 = P.n2, n3 = P.n3;
    if (frozen(P.status, kstep(P) + 1)) return;
    const double *in = part + (size_t)pb * S * 23;
    if (pb < n3) {
        if (!do_moments || c >= 23) return;
        double s = 0.0;
        for (int u = 0; u < S; u++) s += in[(size_t)u * 23 + c];
        const double nxy = (double)(n1 * n2);
        double *out;
        if (c < 7) out = P.stat + (size_t)c * n3;
        else if (c < 14) out = P.stat + (size_t)7 * n3 + (size_t)(c - 7) * n3;
        else out = P.stat + (size_t)14 * n3 + (size_t)(c - 14) * n3;
        const double val = s / nxy;
        out[pb] = val;
        if (P.acc_on) P.tacc[(out - P.stat) + pb] += val;
        return;
    }
    if (!do_tau || c != 0) return;
    const int wall = pb - n3;
    double s = 0.0;
    for (int u = 0; u < S; u++) s += in[(size_t)u * 23];
    const double val = s / (double)((n1 - 2) * (n2 - 2));
    P.stat[(size_t)23 * n3 + wall] = val;
    if (P.acc_on) P.tacc[(size_t)23 * n3 + wall] += val;
}

__global__ void k_stats_fin(const KParams P, int do_moments, int do_tau, int S, const double *part)
{
    grid_dep_enter();
    stats_fin_body(P, do_moments, do_tau, S, part, blockIdx.x, threadIdx.x);
}

// ---------------------------------------------------------------------------
// Diagnostics series (main_v1.9.f90:799-906), every `every` steps:
//   KE = sum over all stored points of (u^2+v^2)+w^2, divided by nP1*nP2*nP3;
//   bulk rho, u and rho*u through the x-planes i = plane(n): over the cells
//   j=1..nP2-1, k=1..nP3-1 the mean of the four corner values times
//   dAyz = dy*(x3(k+1)-x3(k)), summed and divided by Ayz = x3(nP3)*x2(nP2).
// A plane outside 3..nP1-2 gives 0 (the single-rank form of the reference's
// plane(i) > bn(1) .and. plane(i) < en(1) test).  Record layout:
//   [nstep, time, KE, rho_b[np], U_b[np], rhoU_b[np]]
// nstep is -1 when a blow-up stopped the run before that step's diagnostics.
constexpr int kDiagMaxPlanes = 8;

struct DiagParams {
    int nplanes;
    int planes[kDiagMaxPlanes];
    const double *x3q;   // x3 as the diagnostics see it (the deck's F10.6 column after a restart)
    double dy, Ayz;
    int split;           // blocks per plane of the KE sums
    double *part;        // partial sums: KE [nP3][split], then the x-planes' [nplanes][3][nP3]
};

// Partial sums.  Block (k, y): y < split: the KE sum of a share of plane k; then the sums of
// rho, u and rho*u over the cells between planes k and k+1 of x-plane y - split.  One block
// per plane and one per x-plane quantity (each over all cells) left the chip idle: 73 us at
// 101x75x83 with five x-planes, 10 us so split.
__global__ void __launch_bounds__(kStatThreads) k_diag_part(const KParams P, const double *q, const DiagParams D)
{
    __shared__ double red[kStatThreads / 32][3];
    grid_dep_enter();
    const int n1 = P.n1, n2 = P.n2, n3 = P.n3;
    const int k = blockIdx.x + 1, y = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (frozen(P.status, kstep(P) + 1)) return;
    double acc[3] = {0.0, 0.0, 0.0};
    const int m = y - D.split;
    if (m < 0) {
        const unsigned np = (unsigned)n1 * n2;
        for (unsigned p = y * kStatThreads + tid; p < np; p += D.split * kStatThreads) {
            const int jj = (int)(p / (unsigned)n1), ii = (int)(p - (unsigned)jj * n1);
            double x[7];
            ref_var(P, q, ii + 1, jj + 1, k, x);
            acc[0] += (x[1] * x[1] + x[2] * x[2]) + x[3] * x[3];
        }
    } else if (D.planes[m] > 2 && D.planes[m] < n1 - 1 && k < n3) {
        const int ip = D.planes[m];
        const double dAyz = D.dy * (D.x3q[k] - D.x3q[k - 1]);
        for (int j = 1 + tid; j < n2; j += kStatThreads) {
            double a[7], bb[7], cc[7], d[7];
            ref_var(P, q, ip, j, k, a);
            ref_var(P, q, ip, j + 1, k, bb);
            ref_var(P, q, ip, j, k + 1, cc);
            ref_var(P, q, ip, j + 1, k + 1, d);
            acc[0] += (0.25 * (((a[0] + bb[0]) + cc[0]) + d[0])) * dAyz;
            acc[1] += (0.25 * (((a[1] + bb[1]) + cc[1]) + d[1])) * dAyz;
            acc[2] += (0.25 * (((a[0] * a[1] + bb[0] * bb[1]) + cc[0] * cc[1]) + d[0] * d[1])) * dAyz;
        }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const double s = warp_sum(acc[c]);
        if (lane == 0) red[warp][c] = s;
    }
    __syncthreads();
    if (tid < (m < 0 ? 1 : 3)) {
        double t = 0.0;
        for (int w = 0; w < kStatThreads / 32; w++) t += red[w][tid];
        D.part[m < 0 ? (k - 1) * D.split + y : n3 * D.split + (3 * m + tid) * n3 + k - 1] = t;
    }
}

// block 0: KE from the partial sums; block 1+n*np+m: quantity n at plane m.  One warp each.
__global__ void k_diag_fin(const KParams P, const DiagParams D, double *rec, double time)
{
    grid_dep_enter();
    const int n3 = P.n3, b = blockIdx.x, lane = threadIdx.x;
    if (frozen(P.status, kstep(P) + 1)) {
        if (b == 0 && lane == 0) rec[0] = -1.0;
        return;
    }
    const int qn = (b - 1) / max(D.nplanes, 1), m = (b - 1) - qn * D.nplanes;
    const double *in = b == 0 ? D.part : D.part + (size_t)n3 * D.split + (size_t)(3 * m + qn) * n3;
    double t = 0.0;
    for (int e = lane; e < (b == 0 ? n3 * D.split : n3); e += 32) t += in[e];
    t = warp_sum(t);
    if (lane != 0) return;
    if (b == 0) {
        rec[0] = (double)kstep(P);
        rec[1] = time;
        rec[2] = t / ((double)P.n1 * (double)P.n2 * (double)n3);
    } else {
        rec[3 + qn * D.nplanes + m] = t / D.Ayz;
    }
}

// Q-criterion of a velocity field (qInvariant.f90:26-81): central differences
// on the non-uniform coordinates x, y, z; Q = (P^2 - sum S^2 + sum R^2)/2 with
// P = -trace(J), S and R the symmetric and antisymmetric parts of J.  Points
// on the box faces get 0.  u, v, w and Q are [k][j][i].
__global__ void k_qcrit(int n1, int n2, int n3, const double *u, const double *v, const double *w,
                        const double *x, const double *y, const double *z, double *Q)
{
    const unsigned N = (unsigned)n1 * n2 * n3;
    for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) {
        int i, j, k;
        split3(p, n1, n2, i, j, k);
        if (i == 0 || i == n1 - 1 || j == 0 || j == n2 - 1 || k == 0 || k == n3 - 1) {
            Q[p] = 0.0;
            continue;
        }
        const long long si = 1, sj = n1, sk = (long long)n1 * n2;
        const double dx1 = x[i + 1] - x[i], dx2 = x[i] - x[i - 1];
        const double dy1 = y[j + 1] - y[j], dy2 = y[j] - y[j - 1];
        const double dz1 = z[k + 1] - z[k], dz2 = z[k] - z[k - 1];
        const double *U[3] = {u, v, w};
        double J[3][3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double *f = U[c];
            const double f0 = f[p];
            J[c][0] = ((dx2 / dx1) * (f[p + si] - f0) + (dx1 / dx2) * (f0 - f[p - si])) / (dx1 + dx2);
            J[c][1] = ((dy2 / dy1) * (f[p + sj] - f0) + (dy1 / dy2) * (f0 - f[p - sj])) / (dy1 + dy2);
            J[c][2] = ((dz2 / dz1) * (f[p + sk] - f0) + (dz1 / dz2) * (f0 - f[p - sk])) / (dz1 + dz2);
        }
        // sum(S**2) and sum(-R**2) in column-major order
        double as1 = 0.0, as2 = 0.0;
#pragma unroll
        for (int cj = 0; cj < 3; cj++)
#pragma unroll
            for (int ci = 0; ci < 3; ci++) {
                const double sv = ci == cj ? J[ci][ci] : 0.5 * (J[ci][cj] + J[cj][ci]);
                const double rv = ci == cj ? 0.0 : 0.5 * (J[ci][cj] - J[cj][ci]);
                as1 += sv * sv;
                as2 += -(rv * rv);
            }
        const double P_ = -((J[0][0] + J[1][1]) + J[2][2]);
        Q[p] = 0.5 * ((P_ * P_ - as1) - as2);
    }
}

// ---------------------------------------------------------------------------
// Upload: var(1:nP1,1:nP2,1:nP3,1:7) (device copy, [m][k][j][i]) -> state.
// initSolV (main_v1.9.f90:284-294): Q = rho*(1,u,v,w,E) at every point.
__global__ void k_upload(const KParams P, const double *var, const double *cor, double *qa, double *qb, double *qc, double *cs)
{
    const int n1 = P.n1, n2 = P.n2, n3 = P.n3;
    const unsigned N = (unsigned)n1 * n2 * n3;
    for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) {
        int ii, jj, kk;
        split3(p, n1, n2, ii, jj, kk);
        const int i = ii + 1, j = jj + 1, k = kk + 1;
        // T and p (columns 5, 6) are read only on the wall planes, and on the corner
        // columns from cor [2][4][nP3]: the upload copies no others
        const bool wall = (k == 1 || k == n3), corner = (i == 1 || i == n1) && (j == 1 || j == n2);
        double x[7];
#pragma unroll
        for (int m = 0; m < 5; m++) x[m] = var[(size_t)m * N + p];
        const double *co = cor + (size_t)((i == 1 ? 0 : 1) + (j == 1 ? 0 : 2)) * n3 + kk;
        x[5] = wall ? var[(size_t)5 * N + p] : (corner ? co[0] : 0.0);
        x[6] = wall ? var[(size_t)6 * N + p] : (corner ? co[4 * n3] : 0.0);
        const long long o = (long long)k * P.plane + (long long)j * P.px + i;
        double q[5] = {x[0], x[0] * x[1], x[0] * x[2], x[0] * x[3], x[0] * x[4]};
#pragma unroll
        for (int c = 0; c < 5; c++) qa[c * P.vol + o] = q[c];
        if (k == 1 || k == n3) {
#pragma unroll
            for (int c = 0; c < 5; c++) {
                qb[c * P.vol + o] = q[c];
                if (qc) qc[c * P.vol + o] = q[c];
            }
            double *W = P.wp + (size_t)(k == 1 ? 0 : 8) * P.plane + (long long)j * P.px + i;
#pragma unroll
            for (int m = 0; m < 7; m++) W[(size_t)m * P.plane] = x[m];
            W[(size_t)7 * P.plane] = pow(x[5], 0.7);
        } else if ((i == 1 || i == n1) && (j == 1 || j == n2)) {
            const int c = (i == 1 ? 0 : 1) + (j == 1 ? 0 : 2);
#pragma unroll
            for (int m = 0; m < 7; m++) cs[((size_t)k * 4 + c) * 7 + m] = x[m];
        }
    }
}

// periodic images of Q for interior planes (the reference's initial share2P,
// including corner images so every periodic read is consistent); and of the
// wall planes' primitive ring i,j in {0, nP+1}

__global__ void k_fill_ghosts(const KParams P, double *q)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = 2 + blockIdx.z;
    const int n1 = P.n1, n2 = P.n2;
    if (i > n1 + 1 || j > n2 + 1) return;
    const int si = wrap_idx(i, n1), sj = wrap_idx(j, n2);
    if (si == i && sj == j) return;
    const long long o = (long long)k * P.plane + (long long)j * P.px + i;
    const long long s = (long long)k * P.plane + (long long)sj * P.px + si;
#pragma unroll
    for (int c = 0; c < 5; c++) q[c * P.vol + o] = q[c * P.vol + s];
}

__global__ void k_fill_wall_ring(const KParams P)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int wall = blockIdx.z;
    const int n1 = P.n1, n2 = P.n2;
    if (i > n1 + 1 || j > n2 + 1) return;
    if (i >= 1 && i <= n1 && j >= 1 && j <= n2) return;
    const int si = (i == 0 || i == n1 + 1) ? wrap_idx(i, n1) : i;
    const int sj = (j == 0 || j == n2 + 1) ? wrap_idx(j, n2) : j;
    double *W = P.wp + (size_t)wall * 8 * P.plane;
#pragma unroll
    for (int m = 0; m < 8; m++)
        W[(size_t)m * P.plane + (long long)j * P.px + i] = W[(size_t)m * P.plane + (long long)sj * P.px + si];
}

// Download: state -> var(1:nP1,1:nP2,1:nP3,1:7) ([m][k][j][i]); with mean [7][nP3] the
// fluctuation field var(i,j,k,:) - mean(k,:) instead (fluc.f90:63-69)
__global__ void k_download(const KParams P, const double *q, double *var, const double *mean)
{
    const int n1 = P.n1, n2 = P.n2, n3 = P.n3;
    const unsigned N = (unsigned)n1 * n2 * n3;
    for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) {
        int ii, jj, kk;
        split3(p, n1, n2, ii, jj, kk);
        double x[7];
        ref_var(P, q, ii + 1, jj + 1, kk + 1, x);
#pragma unroll
        for (int m = 0; m < 7; m++) var[(size_t)m * N + p] = mean ? x[m] - mean[(size_t)m * n3 + kk] : x[m];
    }
}

// checkSoln over every point (main_v1.9.f90:729-740)
__global__ void k_check(const KParams P, const double *q)
{
    const int n1 = P.n1, n2 = P.n2, n3 = P.n3;
    const unsigned N = (unsigned)n1 * n2 * n3;
    for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) {
        int ii, jj, kk;
        split3(p, n1, n2, ii, jj, kk);
        double x[7];
        ref_var(P, q, ii + 1, jj + 1, kk + 1, x);
        if (x[0] < 0.0 || x[5] < 0.0) flag_blown(P.status, ii + 1, jj + 1, kk + 1, kstep(P));
    }
}

// ---------------------------------------------------------------------------
// Learned subgrid closure: features, filtered-DNS targets, and the closure
// source.  No reference counterpart (the reference resolves every scale).

constexpr int kSgsIn = 13, kSgsOut = 9;   // closure features and fluxes per point

// periodic image of any x or spanwise index on the unique points 2..n-1
__device__ __forceinline__ int wrap_any(int i, int n)
{
    if (i >= 2 && i <= n - 1) return i;
    const int m = n - 2;
    if (i >= 2 - m && i < 2) return i + m;
    if (i > n - 1 && i <= n - 1 + m) return i - m;
    int r = (i - 2) % m;
    if (r < 0) r += m;
    return r + 2;
}

// primitives (rho, u, v, w, T) at (i, j, k): the wall-plane ring on the
// walls, the conservative state elsewhere (exact divisions).  The source is
// selected, not branched to, so that the loads of several points overlap.
__device__ __forceinline__ void prim_at(const KParams &P, const double *q, int i, int j, int k, double x[5])
{
    i = wrap_any(i, P.n1);
    j = wrap_any(j, P.n2);
    const bool wall = k <= 1 || k >= P.n3;
    const long long col = (long long)j * P.px + i, vs = wall ? P.plane : P.vol;
    const double *a = wall ? P.wp + (size_t)(k <= 1 ? 0 : 8) * P.plane + col : q + (long long)k * P.plane + col;
    const double c0 = a[0], c1 = a[vs], c2 = a[2 * vs], c3 = a[3 * vs], c4 = a[(wall ? 5 : 4) * vs];
    const double ri = wall ? 1.0 : 1.0 / c0;
    x[0] = c0;
    x[1] = c1 * ri;
    x[2] = c2 * ri;
    x[3] = c3 * ri;
    x[4] = wall ? c4 : c4 * ri - P.ggMh * ((x[1] * x[1] + x[2] * x[2]) + x[3] * x[3]);
}

// Favre-filtered (rho, u, v, w, T) at (i, j, k): a box of width fw (even)
// in x and spanwise, the trapezoid weights (1/2, 1, .., 1, 1/2) / fw per
// direction; fw = 0 returns the point's own values.  With prod != 0 it also
// returns the filtered rho*u_a*u_b (uu, vv, ww, uv, uw, vw) and rho*u_b*T.
__device__ __forceinline__ void favre_at(const KParams &P, const double *q, int i, int j, int k, int fw,
                                         double f[5], double *prod)
{
    if (fw == 0) {
        prim_at(P, q, i, j, k, f);
        if (prod) {
            const double r = f[0], u = f[1], v = f[2], w = f[3], T = f[4];
            prod[0] = r * u * u; prod[1] = r * v * v; prod[2] = r * w * w;
            prod[3] = r * u * v; prod[4] = r * u * w; prod[5] = r * v * w;
            prod[6] = r * u * T; prod[7] = r * v * T; prod[8] = r * w * T;
        }
        return;
    }
    const int h = fw / 2;
    double sr = 0, su = 0, sv = 0, sw = 0, sT = 0, sp[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int b = -h; b <= h; b++) {
        const double wb = (b == -h || b == h) ? 0.5 : 1.0;
        for (int a = -h; a <= h; a++) {
            const double wgt = wb * ((a == -h || a == h) ? 0.5 : 1.0);
            double x[5];
            prim_at(P, q, i + a, j + b, k, x);
            const double r = x[0], u = x[1], v = x[2], w = x[3], T = x[4], rw = wgt * r;
            sr += wgt * r; su += rw * u; sv += rw * v; sw += rw * w; sT += rw * T;
            if (prod) {
                sp[0] += rw * u * u; sp[1] += rw * v * v; sp[2] += rw * w * w;
                sp[3] += rw * u * v; sp[4] += rw * u * w; sp[5] += rw * v * w;
                sp[6] += rw * u * T; sp[7] += rw * v * T; sp[8] += rw * w * T;
            }
        }
    }
    const double nrm = 1.0 / ((double)fw * (double)fw);
    f[0] = sr * nrm;
    f[1] = su / sr; f[2] = sv / sr; f[3] = sw / sr; f[4] = sT / sr;
    if (prod)
        for (int c = 0; c < 9; c++) prod[c] = sp[c] * nrm;
}

struct SgsSampling {
    int sx, sy, sz, fw;          // gradient strides, filter width
    int i0, ni, j0, nj, k0, nk;  // sample points i0 + sx*a (a < ni), j0 + sy*b, k0 + sz*c
    const double *x3;            // x3(1..nP3) at x3[k-1]
    float *X, *T;                // [n][13], [n][9] (T may be null)
    bool soa;                    // X as [13][n] instead (the closure run's layout)
};

// Favre-filtered (rho, u, v, w, T) at the sample points and the ring around them (their
// gradient neighbours): F [5][nk+2][nj+2][ni+2]; at the sample points also the subgrid
// fluxes T.  Each filtered value is formed once: at every sample point and its six
// neighbours it was formed seven times (256x192x97, strides 4, 3, 3, width 4: 187 us for
// the samples, now 43 + 12 for the features below).
__global__ void __launch_bounds__(128) k_sgs_filter(const KParams P, const double *q, const SgsSampling S, double *F)
{
    const int e1 = S.ni + 2, e2 = S.nj + 2;
    const unsigned ne = (unsigned)e1 * e2 * (S.nk + 2);
    for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < ne; p += gridDim.x * blockDim.x) {
        int a, b, c;
        split3(p, e1, e2, a, b, c);
        const int k = min(max(S.k0 + S.sz * (c - 1), 1), P.n3);
        const bool own = a >= 1 && a <= S.ni && b >= 1 && b <= S.nj && c >= 1 && c <= S.nk;
        double f[5], prod[9];
        favre_at(P, q, S.i0 + S.sx * (a - 1), S.j0 + S.sy * (b - 1), k, S.fw, f, own ? prod : nullptr);
#pragma unroll
        for (int m = 0; m < 5; m++) F[(size_t)m * ne + p] = f[m];
        if (own) {
            const double r = f[0], u = f[1], v = f[2], w = f[3], T = f[4];
            float *Tg = S.T + (((size_t)(c - 1) * S.nj + (b - 1)) * S.ni + (a - 1)) * 9;
            Tg[0] = (float)(prod[0] - r * u * u);
            Tg[1] = (float)(prod[1] - r * v * v);
            Tg[2] = (float)(prod[2] - r * w * w);
            Tg[3] = (float)(prod[3] - r * u * v);
            Tg[4] = (float)(prod[4] - r * u * w);
            Tg[5] = (float)(prod[5] - r * v * w);
            Tg[6] = (float)(prod[6] - r * u * T);
            Tg[7] = (float)(prod[7] - r * v * T);
            Tg[8] = (float)(prod[8] - r * w * T);
        }
    }
}

// Features at every sample point, from the filtered fields F of k_sgs_filter
// (FILTERED; q = F) or the state itself (q).  Gradients by central differences at the
// sample strides (the coarse grid's spacing); y+ from the wall shear of the last
// statistics step.
template <bool FILTERED>
__global__ void __launch_bounds__(128) k_sgs_features(const KParams P, const double *q, const SgsSampling S)
{
    grid_dep_enter();
    const unsigned n = (unsigned)S.ni * S.nj * S.nk;
    const size_t e1 = S.ni + 2, e12 = e1 * (S.nj + 2), ne = e12 * (S.nk + 2);
    const double Lx = 1.0 / P.invdx, Ly = 1.0 / P.invdy;   // dx, dy
    const int n3 = P.n3;
    const double tw = 0.5 * (P.stat[23 * n3] - P.stat[23 * n3 + 1]);
    const double rw = 0.5 * (P.stat[0] + P.stat[n3 - 1]);
    // before the first statistics step the sums are zero: y+ is then 0
    const double ut = rw > 0.0 ? sqrt(fmax(tw, 0.0) / rw) : 0.0, muw = 0.5 * (P.muwb + P.muwt);
    const double cx = 1.0 / (2.0 * S.sx * Lx), cy = 1.0 / (2.0 * S.sy * Ly);
    for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        int a, b, c;
        split3(s, S.ni, S.nj, a, b, c);
        const int i = S.i0 + S.sx * a, j = S.j0 + S.sy * b, k = S.k0 + S.sz * c;
        const int kp = min(k + S.sz, n3), km = max(k - S.sz, 1);
        auto at = [&](int da, int db, int dc, double x[5]) {
            if (FILTERED) {
                const double *f = q + (c + 1 + dc) * e12 + (b + 1 + db) * e1 + (a + 1 + da);
#pragma unroll
                for (int m = 1; m < 5; m++) x[m] = f[m * ne];
            } else {
                prim_at(P, q, i + da * S.sx, j + db * S.sy, dc > 0 ? kp : (dc < 0 ? km : k), x);
            }
        };
        double fxp[5], fxm[5], fyp[5], fym[5], fzp[5], fzm[5];
        at(1, 0, 0, fxp);
        at(-1, 0, 0, fxm);
        at(0, 1, 0, fyp);
        at(0, -1, 0, fym);
        at(0, 0, 1, fzp);
        at(0, 0, -1, fzm);
        const double cz = 1.0 / (S.x3[kp - 1] - S.x3[km - 1]);
        float *X = S.soa ? S.X + s : S.X + (size_t)s * 13;
        const size_t xc = S.soa ? n : 1;
        // du_a/dx_b, a = u, v, w (fields 1..3), b = x, spanwise, wall-normal; then dT/dx_b
#pragma unroll
        for (int m = 0; m < 4; m++) {
            X[(3 * m + 0) * xc] = (float)((fxp[m + 1] - fxm[m + 1]) * cx);
            X[(3 * m + 1) * xc] = (float)((fyp[m + 1] - fym[m + 1]) * cy);
            X[(3 * m + 2) * xc] = (float)((fzp[m + 1] - fzm[m + 1]) * cz);
        }
        const double d = fmin(S.x3[k - 1] - S.x3[0], S.x3[n3 - 1] - S.x3[k - 1]);
        X[12 * xc] = (float)(rw * ut * d * (1.0 / P.invRe) / muw);
    }
}

// Closure source at the interior points from the subgrid fluxes Y [9][n]
// (n = (n1-2)(n2-2)(n3-2), index ((k-2)(n2-2) + (j-2))(n1-2) + i-2; zero on
// the walls): S(rho u_a) = -d tau_ab / dx_b, S(rho E) = -gama d q_b / dx_b
// (the enthalpy flux gama*rho*u*T of the reference's energy equation).
// Streams 36 bytes in and 32 out a point; with wrapped indices formed per access and 64-bit
// quotients it took 27 us at 64x64x65, now 7.
__global__ void k_sgs_div(const KParams P, const float *Y, double gama, double *S)
{
    grid_dep_enter();
    const int n1 = P.n1, n2 = P.n2, n3 = P.n3, m1 = n1 - 2, m2 = n2 - 2;
    const unsigned n = (unsigned)m1 * m2 * (n3 - 2);
    // flux component of (row a, direction b): tau_ab, or q_b for the energy row
    const auto comp = [](int a, int b) { return a == 3 ? 6 + b : (a == b ? a : 2 + a + b); };
    for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        int ii, jj, kk;
        split3(s, m1, m2, ii, jj, kk);
        const double cz = P.czh[kk + 2];
        const unsigned pl = (unsigned)m1 * m2;
        const unsigned xp = ii == m1 - 1 ? s - (m1 - 1) : s + 1, xm = ii == 0 ? s + (m1 - 1) : s - 1;
        const unsigned yp = jj == m2 - 1 ? s - (pl - m1) : s + m1, ym = jj == 0 ? s + (pl - m1) : s - m1;
        const bool top = kk == n3 - 3, bot = kk == 0;   // the fluxes vanish on the walls
        const unsigned zp = top ? s : s + pl, zm = bot ? s : s - pl;
#pragma unroll
        for (int a = 0; a < 4; a++) {
            const float *Yx = Y + (size_t)comp(a, 0) * n, *Yy = Y + (size_t)comp(a, 1) * n, *Yz = Y + (size_t)comp(a, 2) * n;
            const double d = ((double)Yx[xp] - (double)Yx[xm]) * P.hdx + ((double)Yy[yp] - (double)Yy[ym]) * P.hdy +
                             ((top ? 0.0 : (double)Yz[zp]) - (bot ? 0.0 : (double)Yz[zm])) * cz;
            S[(size_t)a * n + s] = a < 3 ? -d : -gama * d;
        }
    }
}

// q_out += cdt * S at the interior rows, their periodic images in x included (those
// in y follow with the wall kernel's image blocks)
__global__ void k_sgs_apply(const KParams P, double *qo, const double *S, double cdt)
{
    grid_dep_enter();
    const int n1 = P.n1, m1 = n1 - 2, m2 = P.n2 - 2, w = n1 + 2;
    const unsigned n = (unsigned)m1 * m2 * (P.n3 - 2), tot = (unsigned)w * m2 * (P.n3 - 2);
    for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < tot; s += gridDim.x * blockDim.x) {
        int i, jj, kk;
        split3(s, w, m2, i, jj, kk);
        const unsigned src = (unsigned)(kk * m2 + jj) * m1 + (wrap_any(i, n1) - 2);
        const long long o = (long long)(kk + 2) * P.plane + (long long)(jj + 2) * P.px + i;
        // S rows: rho*u, rho*v, rho*w, rho*E (state variables 1..4)
#pragma unroll
        for (int a = 0; a < 4; a++) qo[o + (a + 1) * P.vol] += cdt * S[(size_t)a * n + src];
    }
}

// start of a step in a graph replay: step += 1, time += dt (the host's order)
__global__ void k_clock_advance(DevClock *clk, double dt)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        clk->step = clk->step + 1;
        clk->time = clk->time + dt;
    }
}

// double -> float copy (seeds the mixed-precision stage buffers)
__global__ void k_to_float(const double *a, float *b, long long n)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

// self-test of pow07 against the CUDA math library's pow (diagnostics only)
__global__ void k_selftest_pow07(const double *T, double *mine, double *libm, long long n)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        mine[i] = pow07(T[i]);
        libm[i] = pow(T[i], 0.7);
    }
}

// ---------------------------------------------------------------------------
// Persistent ensemble kernel.
//
// One launch runs a block of L time steps of every member of an ensemble.  The
// host lays the work out as phases -- for each member and step: the clock
// advance, then per RK stage the stage kernel's CTAs and the wall kernel's
// blocks, then on statistics steps the two statistics passes -- each phase a
// number of units (one unit = one CTA's work of the kernel it replaces), and
// lists all units of all members in one work list, members interleaved phase
// by phase.  CTAs take units from the list in order through an atomic
// counter.  A unit may start once its member has completed every unit of its
// earlier phases: the member's completion counter reaches the phase's `need`.
// Units are taken in list order and a unit only waits for units earlier in the
// list, which running CTAs hold, so the launch always progresses; each wait is
// still bounded (about a second), after which the CTA records the error and
// stops.
// Every member's arithmetic is the stand-alone kernels' code, so its results
// are bit for bit those of chan_step.
enum PKind { kPClock = 0, kPStage = 1, kPWall = 2, kPStatsPart = 3, kPStatsFin = 4 };

struct PPhase {
    int member;
    int kind;            // PKind
    int variant;         // stage: 0 FP64, 1..3 mixed first / middle / last; wall: 0 double, 1 float state
    int tile;            // stage: CHAN_TILE_32x8 (0) or CHAN_TILE_16x16 (2)
    int nx, ny;          // stage: tiles in x, y; wall: blocks in x, y; stats: blocks per plane (S)
    int kp;              // index of the member's KParams record for this phase
    int units;
    int group;           // wall: wall blocks per unit (the blocks are short)
    unsigned long long need;    // member's completed units before this phase may start
    double dt;                  // clock advance
    const CUtensorMap *tm;      // stage: tensor map of the input buffer
    const CUtensorMap *tmb;     // stage: tensor map of the RK base by tile
    const double *q;            // statistics: the state buffer
    double *part;               // statistics: partial sums
};

struct PItem {
    int phase;
    int unit;
};

// The members' parameter records of the running persistent block, in constant
// memory: a stage body reads its record's fields many times, and from the
// constant cache those reads are cheap where global memory would put a load
// and its latency on each.  A block's graph copies its records here first.
constexpr int kEnsKps = 64;
__constant__ KParams c_ens_kps[kEnsKps];

struct PPlan {
    const PPhase *phases;
    const PItem *items;         // the work list: members' units interleaved phase by phase
    long long nitems;
    unsigned long long *done;   // [members] completed units
    unsigned long long *next;   // work-list position
    int *err;                   // 1: a dependency wait gave up
    DevClock *clk;              // [members]
#ifdef CHAN_PERSIST_GLOBAL_KPS
    const KParams *kps;
#endif
};

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

constexpr unsigned long long kDepWaitNs = 1000000000ull;

template <int TI, int TJ, typename QI, typename QO, typename R>
__device__ __forceinline__ void pstage(const PPhase &F, const KParams &P, int unit, int tid, unsigned char *smem, int *stuck)
{
    using S = StageShape<TI, TJ, R>;
    const int bx = unit % F.nx, r = unit / F.nx, by = r % F.ny, bz = r / F.ny;
    stage_body<TI, TJ, QI, QO, R, 2, true>(P, F.tm, F.tmb, bx, by, bz, tid % S::TX, tid / S::TX, smem, stuck);
}

template <bool MIXED>
struct PersistShape {
    // threads of a persistent CTA: those of the stage units on the 32x8 and 16x16 tiles
    using R = typename std::conditional<MIXED, float, double>::type;
    static constexpr int NT = StageShape<32, 8, R>::NT;
    static_assert(StageShape<16, 16, R>::NT == NT, "both tiles' units have the same threads");
    // dynamic shared memory: the largest unit's, plus the work-item slot
    static constexpr size_t st = MIXED ? (StageShape<32, 8, float>::bytes > StageShape<16, 16, float>::bytes
                                               ? StageShape<32, 8, float>::bytes
                                               : StageShape<16, 16, float>::bytes)
                                       : (StageShape<32, 8, double>::bytes > StageShape<16, 16, double>::bytes
                                              ? StageShape<32, 8, double>::bytes
                                              : StageShape<16, 16, double>::bytes);
    static constexpr size_t wall = sizeof(double) * 2 * 6 * kWallHY * kWallHX;
    static constexpr size_t body = ((st > wall ? st : wall) + 127) / 128 * 128;
    static constexpr size_t bytes = body + 128;
    static constexpr int minb = 2;
};

template <bool MIXED>
__global__ void __launch_bounds__(PersistShape<MIXED>::NT, PersistShape<MIXED>::minb) k_ensemble(const PPlan plan)
{
    using PS = PersistShape<MIXED>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    long long *s_item = reinterpret_cast<long long *>(smem_raw + PS::body);
    int *s_ok = reinterpret_cast<int *>(s_item + 1);
    int *s_stuck = s_ok + 1;   // a stage's copy may still land in this CTA's shared memory
    const int tid = threadIdx.x;
    if (tid == 0) *s_stuck = 0;
    for (;;) {
        if (tid == 0) {
            // the next unit of the work list; wait (bounded) until its member has
            // completed the units of its earlier phases
            long long it = (long long)atomicAdd(plan.next, 1ull);
            // after an error, or with a copy that may still land here: stop
            if (it < plan.nitems && (*(volatile int *)plan.err || *s_stuck)) it = plan.nitems;
            int ok = 1;
            if (it < plan.nitems) {
                const PPhase &F = plan.phases[plan.items[it].phase];
                const unsigned long long *d = plan.done + F.member;
                if (ld_acquire_u64(d) < F.need) {
                    const unsigned long long t0 = global_ns();
                    while (ld_acquire_u64(d) < F.need) {
                        if (global_ns() - t0 > kDepWaitNs) { ok = 0; break; }
                        __nanosleep(256);
                    }
                }
                if (!ok) atomicExch(plan.err, 1);
            }
            *s_item = it;
            *s_ok = ok;
        }
        __syncthreads();
        const long long it = *s_item;
        const int ok = *s_ok;
        __syncthreads();
        if (it >= plan.nitems || !ok) break;
        const PItem I = plan.items[it];
        const PPhase &F = plan.phases[I.phase];
#ifdef CHAN_PERSIST_GLOBAL_KPS
        const KParams &P = plan.kps[F.kp];   // measurement variant: records in global memory
#else
        const KParams &P = c_ens_kps[F.kp];
#endif
        switch (F.kind) {
        case kPClock:
            if (tid == 0) {
                DevClock *c = plan.clk + F.member;
                c->step = c->step + 1;
                c->time = c->time + F.dt;
            }
            break;
        case kPStage:
            if (!MIXED) {
                if (F.tile == 0) pstage<32, 8, double, double, double>(F, P, I.unit, tid, smem_raw, s_stuck);
                else pstage<16, 16, double, double, double>(F, P, I.unit, tid, smem_raw, s_stuck);
            } else if (F.tile == 0) {
                if (F.variant == 1) pstage<32, 8, double, float, float>(F, P, I.unit, tid, smem_raw, s_stuck);
                else if (F.variant == 2) pstage<32, 8, float, float, float>(F, P, I.unit, tid, smem_raw, s_stuck);
                else pstage<32, 8, float, double, float>(F, P, I.unit, tid, smem_raw, s_stuck);
            } else {
                if (F.variant == 1) pstage<16, 16, double, float, float>(F, P, I.unit, tid, smem_raw, s_stuck);
                else if (F.variant == 2) pstage<16, 16, float, float, float>(F, P, I.unit, tid, smem_raw, s_stuck);
                else pstage<16, 16, float, double, float>(F, P, I.unit, tid, smem_raw, s_stuck);
            }
            break;
        case kPWall: {
            WallStage &sp = *reinterpret_cast<WallStage *>(smem_raw);
            const int nb = edge_blocks(P.n1, P.n2, P.n3), b0 = I.unit * F.group, b1 = min(b0 + F.group, nb);
            for (int b = b0; b < b1; b++) {
                if (b > b0) __syncthreads();   // the staging area is reused
                if (F.variant == 0) edge_body<double, PS::NT>(P, b, tid, sp);
                else edge_body<float, PS::NT>(P, b, tid, sp);
            }
            break;
        }
        case kPStatsPart:
            stats_part_body<PS::NT>(P, F.q, 1, 1, F.nx, F.part, I.unit, tid, *reinterpret_cast<StatRed *>(smem_raw));
            break;
        case kPStatsFin: {
            for (int w = tid >> 5; w < 8; w += PS::NT / 32) {
                const int pb = I.unit * 8 + w;
                if (pb < P.n3 + 2) stats_fin_body(P, 1, 1, F.nx, F.part, pb, tid & 31);
            }
            break;
        }
        default:
            break;
        }
        // the unit's writes (all threads) before its completion is counted
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            atomicAdd(plan.done + F.member, 1ull);
        }
    }
}

}  // namespace chan
