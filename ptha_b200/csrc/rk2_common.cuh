// rk2_common.cuh -- device pieces shared by the finite-volume stage kernels
// (rk2.cu: shared-memory tiles; rk2_stream.cu: CTA-wide strips).
#pragma once
#include "swals_kernels.h"

namespace swals {
namespace fv {

// MODE_FLUX: the CFL pass of an adaptive step that also stores every
// cell's dt-independent update terms (CellSums) for the stage-1 update.
enum { MODE_CFL = 0, MODE_STAGE1 = 1, MODE_STAGE2 = 2, MODE_FLUX = 3 };

// Stored per-cell results of a flux pass, everything of update_U that does
// not depend on dt: the flux sums (N - S) + (E - W) of STG, UH, VH (fluxes
// already multiplied by the edge lengths) and the explicit-source sums of
// UH and VH.
template <typename R>
struct CellSums {
    R *d[3];
    double *eu, *ev;
};
enum { FRIC_MANNING = 0, FRIC_CHEZY = 1, FRIC_NONE = 2 };

template <typename R>
struct Rk2Args {
    int nx, ny;
    int64_t P;
    const R *stg, *uh, *vh;        // stage input (U0 for stage 1, U1 for stage 2)
    const R *stg0, *uh0, *vh0;     // backup U0 (stage 2 average)
    R *stg_o, *uh_o, *vh_o;        // stage output
    const R *elv;
    const R *nsq;                  // manning_squared
    R *max_stage;
    Metrics<R> m;
    R theta, half_cfl;
    R lin_fric;                    // linear_friction_coeff
    double dt_fixed;               // used when dt_from_cfl == 0
    int dt_from_cfl;               // stage dt = 1/max(1/maximum_timestep, CFL max) (adaptive)
    double max_dt_inv_init;        // 1/maximum_timestep, rounded to R
    int write_cfl;                 // accumulate the CFL max into sc
    int n_ext;
    int bc_ring;                   // a boundary routine rewrites the outer ring after this stage
    int bext[4];
    R *side;                       // stage-2 pre-average values of the outer two rings
    double *lines;                 // flux_STG on the 4 boundary-flux lines: N[nx], E[ny], S[nx], W[ny]
    DevScalars *sc;
    CellSums<R> cs;                // MODE_FLUX output / stage-1 update input
    int flux_variant;              // FLUX_* bits (compute_fluxes_inner_method)
    R dt_scale;                    // the stage's dt times this (midpoint half step, rk2n last step; else 1)
    int base0;                     // stage 1 updates U0 (stg0..) with this state's fluxes (midpoint)
    R *ev;                         // per-cell eddy viscosity of the stage input (FLUX_EDDY), else null
    R ev_c1, ev_c2;                // eddy_visc_constants
    int pre_bf;                    // stage-1 update: store sc->bf_col0 for the step's two stage boundaries
    BoundaryFn bf;                 // ... of this boundary function, cell-centre x coordinates bf_x
    const R *bf_x;
};

template <typename R> struct Cell { R stg, dep, u, v, elv; };

__device__ __forceinline__ void atomic_max_pos_double(unsigned long long *addr, double v)
{
    atomicMax(addr, (unsigned long long)__double_as_longlong(v));
}

// Whether a and b have the same sign bit.
__device__ __forceinline__ bool same_sign(double a, double b) { return (__double2hiint(a) ^ __double2hiint(b)) >= 0; }
__device__ __forceinline__ bool same_sign(float a, float b) { return (__float_as_int(a) ^ __float_as_int(b)) >= 0; }

// Whether v is +0.
__device__ __forceinline__ bool bits_zero(double v) { return (__double2hiint(v) | __double2loint(v)) == 0; }
__device__ __forceinline__ bool bits_zero(float v) { return __float_as_int(v) == 0; }

// MC limiter, extrapolation_limiting_mod.f90:63-79 (sign(1,a) == copysign),
// as the reference writes it, returning TWICE the limited gradient; the edges
// take U -+ a quarter of it in one fused operation (a product by a power of
// two is exact, but in subnormals, so it rounds as the reference's U -+ 1/2
// gradient does).
template <typename R>
__device__ __forceinline__ R mc_double_gradient_ref(R local, R lower, R upper, R th)
{
    const R a = upper - local;
    const R b = local - lower;
    const R sa = copysign(R(1), a);
    const R sb = copysign(R(1), b);
    const R half_sasb = R(0.5) * (sa + sb);
    const R d = rmin(R(fabs(a)), R(fabs(b))) * half_sasb * th;
    const R e = R(0.5) * (a + b);
    const R c = (d == R(0)) ? R(0) : e;
    return R(2) * ((d > R(0)) ? rmin(c, d) : rmax(c, d));
}

// The same for an ordinary theta (th2 is twice it): zero for different
// signs, else min(|a + b|, min(|a|,|b|) 2 theta) with the sign of a; half the
// instructions.  Infinities and NaNs come out as they do there, a NaN's sign
// included, by which the next step's sign products spread it.
template <typename R>
__device__ __forceinline__ R mc_double_gradient(R local, R lower, R upper, R th2)
{
    const R a = upper - local;
    const R b = local - lower;
    const R fa = R(fabs(a)), fb = R(fabs(b)), e = a + b, fe = R(fabs(e));
    const R d = rmin(fa, fb) * (same_sign(a, b) ? th2 : R(0));
    // (d zero is the answer whatever fe, which a NaN neighbour makes NaN)
    return (d < fe || bits_zero(d)) ? copysign(d, a) : e;
}

// theta_wd of DE1_inner_include.f90:751-757 / :813-819.
template <typename R>
__device__ __forceinline__ R theta_wd(R d0, R d1, R d2, R theta)
{
    const R coef4 = R(1) / (K<R>::limiter_coef2() - K<R>::limiter_coef1());
    const R mindep = rmin(rmin(d0, d1), d2) - K<R>::min_depth();
    const R maxdep = rmax(rmax(d0, d1), d2) + K<R>::limiter_coef3() * K<R>::min_depth();
    const R theta_local = coef4 * (mindep / maxdep - K<R>::limiter_coef1());
    return rmax(theta * rmin(R(1), theta_local), R(0));
}

// Bounds of the least and greatest of three depths (>= 0): for FP64 from
// their high words, whose order as integers is the numbers' own.
__device__ __forceinline__ void depth_bounds(double d0, double d1, double d2, double &lo, double &lo_up, double &hi)
{
    const int h0 = __double2hiint(d0), h1 = __double2hiint(d1), h2 = __double2hiint(d2);
    const int mn = min(min(h0, h1), h2), mx = max(max(h0, h1), h2);
    lo = __hiloint2double(mn, 0);
    lo_up = __hiloint2double(mn, -1);
    hi = __hiloint2double(mx, -1);
}
__device__ __forceinline__ void depth_bounds(float d0, float d1, float d2, float &lo, float &lo_up, float &hi)
{
    lo = lo_up = rmin(rmin(d0, d1), d2);
    hi = rmax(rmax(d0, d1), d2);
}

// Twice the limited gradients of stage, depth, u, v (mc_double_gradient).
template <typename R> struct Grad { R ds, dd, du, dv; };

// The limited gradients of cell c between lo and up.  theta_wd's quotient
// mindep / maxdep matters only between 0.1 (theta 0 below) and 0.3 (theta
// above): everywhere but on steep shallows bounds of the depths, with room
// for their truncation and for rounding, settle it without the division.
// Where they do not (or a depth is not finite), the reference's formulas.
template <typename R>
__device__ __forceinline__ Grad<R> limited(const Cell<R> &cl, const Cell<R> &c, const Cell<R> &cu, R theta)
{
    R lo, lo_up, hi;
    depth_bounds(cl.dep, c.dep, cu.dep, lo, lo_up, hi);
    const R mad = K<R>::min_depth(), wide = K<R>::limiter_coef3() * K<R>::min_depth();
    const bool deep = lo - R(1.001) * mad > R(0.3003) * (hi + R(1.001) * wide);
    const bool shallow = lo_up - R(0.999) * mad < R(0.0998) * (hi + R(0.999) * wide);
    Grad<R> g;
    if (deep || shallow) {
        const R th2 = deep ? R(2) * rmax(theta, R(0)) : R(0);
        g.ds = mc_double_gradient<R>(c.stg, cl.stg, cu.stg, th2);
        g.dd = mc_double_gradient<R>(c.dep, cl.dep, cu.dep, th2);
        g.du = mc_double_gradient<R>(c.u, cl.u, cu.u, th2);
        g.dv = mc_double_gradient<R>(c.v, cl.v, cu.v, th2);
    } else {
        const R th = theta_wd<R>(cl.dep, c.dep, cu.dep, theta);
        g.ds = mc_double_gradient_ref<R>(c.stg, cl.stg, cu.stg, th);
        g.dd = mc_double_gradient_ref<R>(c.dep, cl.dep, cu.dep, th);
        g.du = mc_double_gradient_ref<R>(c.u, cl.u, cu.u, th);
        g.dv = mc_double_gradient_ref<R>(c.v, cl.v, cu.v, th);
    }
    return g;
}

// Stage, depth and velocities reconstructed at an edge of a cell
// (DE1_inner_include.f90's U +- 1/2 gradient; Grad holds twice the gradient).
template <typename R> struct Face { R s, d, u, v; };
template <typename R>
__device__ __forceinline__ Face<R> face_above(const Cell<R> &c, const Grad<R> &g)   // the north or east edge
{
    const R q = R(0.25);
    Face<R> f;
    f.s = fma(q, g.ds, c.stg); f.d = fma(q, g.dd, c.dep); f.u = fma(q, g.du, c.u); f.v = fma(q, g.dv, c.v);
    return f;
}
template <typename R>
__device__ __forceinline__ Face<R> face_below(const Cell<R> &c, const Grad<R> &g)   // the south or west edge
{
    const R q = R(-0.25);
    Face<R> f;
    f.s = fma(q, g.ds, c.stg); f.d = fma(q, g.dd, c.dep); f.u = fma(q, g.du, c.u); f.v = fma(q, g.dv, c.v);
    return f;
}

// What the *_eddyvisc variants add to an edge: the eddy viscosities of the two
// cells, the velocity differences and the distance they are taken over.
template <typename R> struct EddyIn { R ev_n, ev_p, du, dv, vel_div; };

template <typename R>
struct EdgeRes {
    R f[3];          // STG, UH, VH flux (already multiplied by edge length)
    double es_pos;   // explicit-source contribution to the cell on the + side
    double es_neg;   // contribution to the cell on the - side
};

// A momentum flux of the *_eddyvisc variants (DE1_inner_include.f90:
// 289-358, 551-620): the advective part plus the HLL and turbulent
// diffusions, summed unless both have the same sign
// (reduced_numerical_diffusion), when the larger magnitude is taken.
template <typename R>
__device__ __forceinline__ R eddy_momentum_flux(R adv, R hll, R turb)
{
    const R dmax = rmax(R(fabs(turb)), R(fabs(hll)));
    const R tot = (turb * hll > R(0)) ? R(copysign(dmax, turb)) : turb + hll;
    return adv + tot;
}

// One Audusse/HLL edge of DE1_inner_include.f90 (:187-430 NS, :456-716 EW).
// The stage kernels are bound by FP64 issue and latency, so what an edge does
// not need is left out without changing a bit of its result: the square roots
// and the quotient by straight-line sequences (sqrt_ord, div_ord), the Froude
// factor and theta_wd's quotient only where they are not settled by bounds,
// the limiter without sign products.  Measured on the rk2 beach, a step:
// 2048^2 FP64 0.657 -> 0.584 ms, FP32 0.506 -> 0.456, 300 x 200 FP64 0.086 ->
// 0.071; midpoint on a spherical 930^2 patch 0.196 -> 0.167.
// NS=true: normal velocity v, edge between (i,j-1) and (i,j).
// variant: compute_fluxes_inner_method as FLUX_* bits (swals_kernels.h);
// 0 is the default 'DE1_low_fr_diffusion'.  EDDY (FLUX_EDDY): vel_div is
// distance_left_edge(i) for NS edges, the mean of distance_bottom_edge(j),
// (j+1) for EW edges.  n, p: the faces of the two cells at the edge, dep_ and
// elv_ their depths and elevations.
template <typename R, bool NS, bool EDDY = false>
__device__ __forceinline__ void edge_faces(const Face<R> &n, R dep_n, R elv_n, const Face<R> &p, R dep_p, R elv_p,
                                           R edge_len, EdgeRes<R> &out, R &max_speed, int variant = 0,
                                           const EddyIn<R> &eddy = EddyIn<R>())
{
    const R half = R(0.5);
    const double half_gravity = (double)(half * K<R>::gravity());
    const R EPS = R(1.0e-12);
    // sqrt(gravity * minimum_allowed_depth) in the state precision (the
    // correctly rounded root of the rounded product, as written out here)
    const R EPS_gs = sizeof(R) == 8 ? R(0x1.4462fb7ff5035p-7) : R(0x1.4462fcp-7f);
    const R beta = R(1.0);
    // (Sums, differences and products that the reference forms in double from
    // two values of the state precision and rounds to it are formed in the
    // state precision here: with 53 bits against 24 the second rounding
    // changes nothing.)
    const R z_neg = n.s - n.d;
    const R z_pos = p.s - p.d;
    const R z_half = rmax(z_neg, z_pos);

    // a side's depth at the edge is zero exactly where its stage is not above z_half
    const bool dry_neg = z_half >= n.s, dry_pos = z_half >= p.s;
    const R stage_neg_star = dry_neg ? z_half : n.s;
    const R stage_pos_star = dry_pos ? z_half : p.s;
    const R d_neg = stage_neg_star - z_half, d_pos = stage_pos_star - z_half;
    const double depth_neg = (double)n.d, depth_pos = (double)p.d;
    const double depth_neg_star = (double)d_neg, depth_pos_star = (double)d_pos;
    const R u_neg = dry_neg ? R(0) : n.u, v_neg = dry_neg ? R(0) : n.v;
    const R u_pos = dry_pos ? R(0) : p.u, v_pos = dry_pos ? R(0) : p.v;
    const R vel_beta_neg = (NS ? v_neg : u_neg) * beta;
    const R vel_beta_pos = (NS ? v_pos : u_pos) * beta;
    const R tran_neg = NS ? u_neg : v_neg, tran_pos = NS ? u_pos : v_pos;
    const R qn_neg = vel_beta_neg * d_neg, qn_pos = vel_beta_pos * d_pos;
    const R qt_neg = tran_neg * d_neg, qt_pos = tran_pos * d_pos;
    R gs_neg = R(sqrt_ord((double)K<R>::gravity() * depth_neg_star));
    R gs_pos = R(sqrt_ord((double)K<R>::gravity() * depth_pos_star));

    R s_max = rmax(rmax(vel_beta_neg + gs_neg, vel_beta_pos + gs_pos), R(0));
    R s_min = rmin(rmin(vel_beta_neg - gs_neg, vel_beta_pos - gs_pos), R(0));
    double denom = (double)(s_max - s_min);
    double quotient = div_ord((double)edge_len, denom);   // unused where denom is tiny
    const R depth_sum = d_neg + d_pos;
    if (!((double)depth_sum < 1.0e280 && denom < 1.0e280)) {   // a run that has blown up: the plain operators
        gs_neg = R(sqrt((double)K<R>::gravity() * depth_neg_star));
        gs_pos = R(sqrt((double)K<R>::gravity() * depth_pos_star));
        s_max = rmax(rmax(vel_beta_neg + gs_neg, vel_beta_pos + gs_pos), R(0));
        s_min = rmin(rmin(vel_beta_neg - gs_neg, vel_beta_pos - gs_pos), R(0));
        denom = (double)(s_max - s_min);
        quotient = (double)edge_len / denom;
    }
    const double inv_denom = (denom > (double)EPS && (gs_pos > EPS_gs || gs_neg > EPS_gs)) ? quotient : 0.0;
    const R sminsmax = s_min * s_max * R(1);
    // reduced_momentum_diffusion (the low_fr_diffusion variants), else 1:
    // sqrt(max(0.001, min(1, fr2num / fr2den))).  Where the Froude number is
    // low, as in all but shallow or fast water, the bounds below show that the
    // quotient is under 0.001 and the root that of 0.001; only the other
    // edges form it.
    R fr2 = R(1);
    if (!(variant & FLUX_PLAIN_DIFFUSION)) {
        const R num_b = fma(vel_beta_neg, vel_beta_neg,
                            fma(vel_beta_pos, vel_beta_pos, fma(tran_neg, tran_neg, tran_pos * tran_pos)));
        const R den_b = K<R>::gravity() * depth_sum + R(1.0e-10);
        fr2 = sizeof(R) == 8 ? R(0x1.030dc4ea03a72p-5) : R(0x1.030dc6p-5f);
        if (!(num_b < R(0.00099) * den_b)) {
            const R fr2num = ((v_neg * v_neg + v_pos * v_pos) + u_neg * u_neg) + u_pos * u_pos;
            const R fr2den = (gs_neg * gs_neg + gs_pos * gs_pos) + R(1.0e-10);
            fr2 = R(sqrt(rmax(R(0.001), rmin(R(1), fr2num / fr2den))));
        }
        fr2 = beta * fr2;
    }

    const R f_mass = R((double)((s_max * qn_neg - s_min * qn_pos) + sminsmax * (stage_pos_star - stage_neg_star)) *
                       inv_denom);
    R f_norm, f_tran;
    if (!EDDY) {
        f_norm = R((double)((s_max * qn_neg * vel_beta_neg - s_min * qn_pos * vel_beta_pos) +
                            fr2 * sminsmax * (qn_pos - qn_neg)) * inv_denom);
        if (variant & FLUX_UPWIND_TRANSVERSE)   // upwind_transverse_momentum: the transverse velocity upwind of the mass flux
            f_tran = beta * ((f_mass > R(0)) ? tran_neg : tran_pos) * f_mass;
        else
            f_tran = R((double)((s_max * qt_neg * vel_beta_neg - s_min * qt_pos * vel_beta_pos) +
                                fr2 * sminsmax * (qt_pos - qt_neg)) * inv_denom);
    } else {
        // turbulent diffusion: eddy_visc * depth * edge length * velocity gradient,
        // with the geometric mean of the edge depths
        const R evh = half * (eddy.ev_p + eddy.ev_n);
        const R gdep = R(sqrt(depth_neg_star * depth_pos_star));
        R adv = R((double)(s_max * qn_neg * vel_beta_neg - s_min * qn_pos * vel_beta_pos) * inv_denom);
        R hll = R((double)(fr2 * sminsmax * (qn_pos - qn_neg)) * inv_denom);
        R turb = -(evh * gdep * edge_len * ((NS ? eddy.dv : eddy.du) / eddy.vel_div));
        f_norm = eddy_momentum_flux<R>(adv, hll, turb);
        if (variant & FLUX_UPWIND_TRANSVERSE) {
            adv = beta * ((f_mass > R(0)) ? tran_neg : tran_pos) * f_mass;
            hll = R(0);
        } else {
            adv = R((double)(s_max * qt_neg * vel_beta_neg - s_min * qt_pos * vel_beta_pos) * inv_denom);
            hll = R((double)(fr2 * sminsmax * (qt_pos - qt_neg)) * inv_denom);
        }
        turb = -(evh * gdep * edge_len * ((NS ? eddy.du : eddy.dv) / eddy.vel_div));
        f_tran = eddy_momentum_flux<R>(adv, hll, turb);
    }
    out.f[0] = f_mass;
    out.f[1] = NS ? f_tran : f_norm;
    out.f[2] = NS ? f_norm : f_tran;

    const double half_g_hh_edge = inv_denom * half_gravity *
        ((double)s_max * depth_neg_star * depth_neg_star - (double)s_min * depth_pos_star * depth_pos_star);
    const double bs_neg = half_gravity * ((depth_neg_star - depth_neg) * (depth_neg_star + depth_neg) -
                                          (depth_neg + (double)dep_n) * (double)(z_neg - elv_n));
    out.es_neg = bs_neg * (double)edge_len - half_g_hh_edge;
    const double bs_pos = half_gravity * ((depth_pos_star - depth_pos) * (depth_pos_star + depth_pos) -
                                          (depth_pos + (double)dep_p) * (double)(z_pos - elv_p));
    out.es_pos = half_g_hh_edge - bs_pos * (double)edge_len;

    max_speed = rmax(s_max, -s_min);
}

// A speed's candidate for the largest 1/dt of its edge.
template <typename R>
__device__ __forceinline__ double cfl_rate(R max_speed, R dx_cfl_half_inv)
{
    return (max_speed > R(1.0e-12)) ? (double)max_speed * (double)dx_cfl_half_inv : 0.0;
}

// The edge between two cells from their values and (twice the) gradients.
template <typename R, bool NS, bool EDDY = false>
__device__ __forceinline__ void edge_flux(const Cell<R> &cn, const Grad<R> &gn, const Cell<R> &cp, const Grad<R> &gp,
                                          R edge_len, R dx_cfl_half_inv, EdgeRes<R> &out, double &cfl_cand,
                                          int variant = 0, R ev_n = R(0), R ev_p = R(0), R vel_div = R(1))
{
    EddyIn<R> eddy;
    if (EDDY) { eddy.ev_n = ev_n; eddy.ev_p = ev_p; eddy.vel_div = vel_div; eddy.du = cp.u - cn.u; eddy.dv = cp.v - cn.v; }
    R max_speed;
    edge_faces<R, NS, EDDY>(face_above(cn, gn), cn.dep, cn.elv, face_below(cp, gp), cp.dep, cp.elv, edge_len, out,
                            max_speed, variant, eddy);
    cfl_cand = cfl_rate<R>(max_speed, dx_cfl_half_inv);
}

// Timestep of a stage: fixed, or domain%max_dt of the first stage
// 1/max(1/maximum_timestep, max speed/(dx cfl/2)) for adaptive stepping.
template <typename R>
__device__ __forceinline__ R stage_dt(const Rk2Args<R> &a)
{
    if (a.dt_from_cfl) {
        const double bits_max = __longlong_as_double((long long)a.sc->max_dt_inv_bits);
        const R inv = R(fmax(a.max_dt_inv_init, bits_max));
        return (R(1) / inv) * a.dt_scale;
    }
    return R(a.dt_fixed) * a.dt_scale;
}

// The dt-independent part of update_U for cell (i, r)
// (update_U_DE1_inner_include.f90:38-96) from its four edges: the flux sums
// (n_hi - n_lo) + (w_hi - w_lo) and the explicit sources of UH and VH,
// accumulated in the reference's order.  Um_uh / Um_vh are U(i,j,UH/VH)
// after compute_depth_and_velocity (zero where depth <= minimum_allowed_depth);
// only the spherical terms read them.
template <typename R> struct CellFlux {
    R d[3];
    double eu, ev;
};
template <typename R, bool SPH, bool COR>
__device__ __forceinline__ CellFlux<R> cell_flux(const Rk2Args<R> &a, int i, int r, const Cell<R> &c, R Um_uh,
                                                 R Um_vh, const EdgeRes<R> &n_lo, const EdgeRes<R> &n_hi,
                                                 const EdgeRes<R> &w_lo, const EdgeRes<R> &w_hi)
{
    const int nx = a.nx, ny = a.ny;
    CellFlux<R> f;
    f.d[0] = (n_hi.f[0] - n_lo.f[0]) + (w_hi.f[0] - w_lo.f[0]);
    f.d[1] = (n_hi.f[1] - n_lo.f[1]) + (w_hi.f[1] - w_lo.f[1]);
    f.d[2] = (n_hi.f[2] - n_lo.f[2]) + (w_hi.f[2] - w_lo.f[2]);
    double es_uh = 0.0, es_vh = 0.0, es_jm1 = 0.0;
    if (r >= 1) {
        if (i >= 1) {
            es_vh = n_lo.es_pos;   // NS loop (:403-409)
            es_uh = w_lo.es_pos;   // EW loop (:649-654)
            if (SPH) {
                const double dep = (double)c.dep;
                const double hg = (double)(R(0.5) * K<R>::gravity());
                es_vh = es_vh + hg * dep * dep * (double)(a.m.dxb[r + 1] - a.m.dxb[r]);
                if (COR) {
                    const R cm = a.m.area[r] * a.m.cor[r];
                    es_uh = es_uh + (double)(cm * Um_vh);
                    es_vh = es_vh - (double)(cm * Um_uh);
                }
                const R cm2 = a.m.area[r] * a.m.tanlat[r] * c.u;
                es_uh = es_uh + (double)(cm2 * Um_vh);
                es_vh = es_vh - (double)(cm2 * Um_uh);
            }
        }
        es_uh = es_uh + ((i + 1 <= nx - 1) ? w_hi.es_neg : 0.0);  // explicit_source_im1_work (:721)
    }
    if (r + 1 <= ny - 1 && i >= 1) es_jm1 = n_hi.es_neg;          // explicit_source_VH_j_minus_1(i, j+1)
    f.eu = es_uh;
    f.ev = es_vh + es_jm1;
    return f;
}

// U(i,j,UH/VH) after compute_depth_and_velocity: the stage input where the
// fixed-up depth exceeds minimum_allowed_depth, else zero.
template <typename R>
__device__ __forceinline__ void fixed_momenta(const Rk2Args<R> &a, int64_t o, const Cell<R> &c, R &Um_uh, R &Um_vh)
{
    if (c.dep > K<R>::min_depth()) { Um_uh = a.uh[o]; Um_vh = a.vh[o]; }
    else { Um_uh = R(0); Um_vh = R(0); }
}

// The semi-implicit friction factor of cell o of the stage input (1 without friction).
template <typename R, int FRIC>
__device__ __forceinline__ R friction_factor(const Rk2Args<R> &a, R nsq, const Cell<R> &c, R dt)
{
    if (FRIC == FRIC_NONE) return R(1);
    constexpr bool CHEZY = (FRIC == FRIC_CHEZY);
    const R mad = K<R>::min_depth();
    const R depth = c.dep;
    const R speed2 = c.u * c.u + c.v * c.v;
    const R dg = dt * K<R>::gravity() * rmax(depth, R(0));
    const R large = sizeof(R) == 8 ? R(1.0e280) : R(1.0e37);
    if ((double)depth < 1.0e30 && speed2 < large) {
        const R fs = nsq * sqrt_ord(speed2) * R(pow_friction<CHEZY, true>((double)rmax(depth, mad)));
        const R d = (R(1) + dg * fs) + dt * a.lin_fric;
        if (sizeof(R) == 8 || d < large) return rcp_ord(d);
    }
    // a run that has blown up: the plain operators
    const R fs = nsq * R(sqrt(speed2)) * R(pow_friction<CHEZY>((double)rmax(depth, mad)));
    return R(1) / ((R(1) + dg * fs) + dt * a.lin_fric);
}

// Stage 2's U0 and max_stage of a cell: read where they are used, or loaded
// ahead by the caller.
template <typename R> struct Stage2Mem {
    __device__ __forceinline__ R s(const Rk2Args<R> &a, int64_t o) const { return a.stg0[o]; }
    __device__ __forceinline__ R uh(const Rk2Args<R> &a, int64_t o) const { return a.uh0[o]; }
    __device__ __forceinline__ R vh(const Rk2Args<R> &a, int64_t o) const { return a.vh0[o]; }
    __device__ __forceinline__ R mx(const Rk2Args<R> &a, int64_t o) const { return a.max_stage[o]; }
};
template <typename R> struct Stage2Reg {
    R s_, uh_, vh_, mx_;
    __device__ __forceinline__ R s(const Rk2Args<R> &, int64_t) const { return s_; }
    __device__ __forceinline__ R uh(const Rk2Args<R> &, int64_t) const { return uh_; }
    __device__ __forceinline__ R vh(const Rk2Args<R> &, int64_t) const { return vh_; }
    __device__ __forceinline__ R mx(const Rk2Args<R> &, int64_t) const { return mx_; }
};

// The rest of update_U for cell (i, r) with the stage's dt: the flux
// update, the wet/dry test, the semi-implicit friction and the explicit
// sources; stage 2 also forms the rk2 average and max_stage.
// inv_cell_area_dt is the row's dt / area_cell_y(r) (a row constant the
// callers may evaluate once per row); factor() gives the friction factor, in
// gives stage 2's U0 and max_stage of the cell (Stage2Mem, Stage2Reg).
template <typename R, int MODE, typename Factor, typename Stage2>
__device__ __forceinline__ void fv_apply(const Rk2Args<R> &a, int i, int r, const Cell<R> &c, R Um_uh, R Um_vh,
                                         const CellFlux<R> &f, R inv_cell_area_dt, Factor factor, Stage2 in)
{
    const int nx = a.nx, ny = a.ny;
    const int64_t P = a.P;
    const R mad = K<R>::min_depth();
    const int64_t o = (int64_t)r * P + i;
    R U_stg = c.stg;
    R U_uh = Um_uh, U_vh = Um_vh;
    if (MODE == MODE_STAGE1 && a.base0) {
        // one_midpoint_step's full step: U was reset to the backup, and
        // update_U applies the midpoint's fluxes to it.
        U_stg = a.stg0[o]; U_uh = a.uh0[o]; U_vh = a.vh0[o];
    }

    U_stg = U_stg - inv_cell_area_dt * f.d[0];
    U_uh = U_uh - inv_cell_area_dt * f.d[1];
    U_vh = U_vh - inv_cell_area_dt * f.d[2];

    if (U_stg <= c.elv + mad) {
        U_uh = R(0);
        U_vh = R(0);
    } else {
        const R implicit_factor = factor();
        U_uh = R((double)U_uh + (double)inv_cell_area_dt * f.eu);
        U_uh = U_uh * implicit_factor;
        U_vh = R((double)U_vh + (double)inv_cell_area_dt * f.ev);
        U_vh = U_vh * implicit_factor;
    }

    if (MODE == MODE_STAGE2) {
        const bool outer2 = (i <= 1 || i >= nx - 2 || r <= 1 || r >= ny - 2);   // the outer two rings
        if (a.bc_ring && outer2) {
            // Keep the pre-average outer two rings for the boundary kernel.
            R *side = a.side;
            const int cols[4] = {0, 1, nx - 2, nx - 1};
            const int rows[4] = {0, 1, ny - 2, ny - 1};
            for (int k = 0; k < 4; k++) {
                if (i == cols[k]) {
                    R *d = side + ((int64_t)k * ny + r) * 3;
                    d[0] = U_stg; d[1] = U_uh; d[2] = U_vh;
                }
                if (r == rows[k]) {
                    R *d = side + (int64_t)4 * ny * 3 + ((int64_t)k * nx + i) * 3;
                    d[0] = U_stg; d[1] = U_uh; d[2] = U_vh;
                }
            }
        }
        U_stg = R(0.5) * (U_stg + in.s(a, o));
        U_uh = R(0.5) * (U_uh + in.uh(a, o));
        U_vh = R(0.5) * (U_vh + in.vh(a, o));
        if (a.max_stage) {
            const bool ring = a.bc_ring && outer2 && ((i == 0 && a.bext[3]) || (i == nx - 1 && a.bext[1]) ||
                                                      (r == 0 && a.bext[2]) || (r == ny - 1 && a.bext[0]));
            if (!ring) {
                R mx = in.mx(a, o);
                a.max_stage[o] = (U_stg > mx) ? U_stg : mx;
            }
        }
    }
    a.stg_o[o] = U_stg;
    a.uh_o[o] = U_uh;
    a.vh_o[o] = U_vh;
}

// update_U for cell (i, r) (update_U_DE1_inner_include.f90:38-96) from its
// fixed-up centre values and its four edges.
template <typename R, int MODE, bool SPH, bool COR, int FRIC>
__device__ __forceinline__ void fv_update(const Rk2Args<R> &a, int i, int r, const Cell<R> &c, const EdgeRes<R> &n_lo,
                                          const EdgeRes<R> &n_hi, const EdgeRes<R> &w_lo, const EdgeRes<R> &w_hi,
                                          R dt, R inv_cell_area_dt)
{
    R Um_uh, Um_vh;
    fixed_momenta<R>(a, (int64_t)r * a.P + i, c, Um_uh, Um_vh);
    const CellFlux<R> f = cell_flux<R, SPH, COR>(a, i, r, c, Um_uh, Um_vh, n_lo, n_hi, w_lo, w_hi);
    fv_apply<R, MODE>(a, i, r, c, Um_uh, Um_vh, f, inv_cell_area_dt,
                      [&] { return friction_factor<R, FRIC>(a, FRIC == FRIC_NONE ? R(0) : a.nsq[(int64_t)r * a.P + i], c, dt); },
                      Stage2Mem<R>());
}
}  // namespace fv
}  // namespace swals
