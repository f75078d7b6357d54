// rk2_stream.cu -- the finite-volume stage kernel on CTA-wide strips.
//
// Same computation as the shared-memory tile kernel in rk2.cu (and the same
// device functions: limited, edge_faces, cell_flux, fv_apply), organised for
// sm_100a's FP64 pipes:
//   - the SW threads of a CTA own a strip of SW - 4 output columns (the two
//     columns on either side are the limiter's halo) and march down SH rows
//     plus two rows at each end, one column a thread;
//   - shared memory, one array per field, holds what neighbouring columns
//     read (the last three fixed-up rows, the east faces, the west edges) and
//     what a thread keeps for its own next rows (north and west faces, the
//     south edge): in registers these cost a CTA an SM;
//   - each edge, gradient and face is formed once; two barriers a row;
//   - the next row's loads are issued before the current row is processed,
//     the lines that only the update reads are started towards L2, and stage 2
//     loads them a barrier ahead.
// Bound by instruction issue: 2048^2 FP64 stage 2 250 us, 1455 thread
// instructions a cell, 72 % of the issue slots, FP64 pipe 49 % busy; the flux
// pass 205 us, 1095, 68 %, 50 % (1792 and 1523 instructions, 315 and 263 us,
// before the straight-line roots and quotients and the sign-free limiter).
#include "rk2_common.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

namespace swals {
namespace {
using namespace fv;

constexpr unsigned FULL = 0xffffffffu;
constexpr int SW = 128;         // threads of a strip (and of a CTA)
constexpr int SO = SW - 4;      // its output columns
constexpr int RC = 64;          // segments of up to this many rows keep their row constants in shared memory

template <typename R> struct Raw { R s, uh, vh, e; };

// compute_depth_and_velocity for one cell (domain_mod.f90:1387-1412).
template <typename R>
__device__ __forceinline__ Cell<R> fix_up(const Raw<R> &x, bool valid, bool &fixed)
{
    Cell<R> c;
    c.stg = R(0); c.dep = R(0); c.u = R(0); c.v = R(0); c.elv = R(0);
    fixed = false;
    if (valid) {
        R s = x.s;
        const R e = x.e;
        R dep = s - e;
        if (dep > K<R>::min_depth()) {
            const R depth_inv = depth_inverse(dep);
            c.u = x.uh * depth_inv;
            c.v = x.vh * depth_inv;
        } else if (dep < R(0)) {
            dep = R(0);
            s = e;
            fixed = true;
        }
        c.stg = s; c.dep = dep; c.elv = e;
    }
    return c;
}

// Bring a line into L2 ahead of its use (no register is written).
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// What the threads of a strip share, one array per field, with a column of
// padding either side (read by the outermost threads, whose results nothing
// uses).
template <typename R>
struct Strip {
    R stg[3][SW + 2], dep[3][SW + 2], u[3][SW + 2], v[3][SW + 2], elv[3][SW + 2];   // fixed-up rows r, r-1, r-2
    R fs[2][SW + 2], fd[2][SW + 2], fu[2][SW + 2], fv[2][SW + 2];                   // east faces of rows r-1, r-2
    R f0[SW + 2], f1[SW + 2], f2[SW + 2];                                           // west edges of row r-2
    double es[SW + 2];
    // a thread's own: the north and west faces and the south edge of row r-2
    R ns[SW], nd[SW], nu[SW], nv[SW];
    R ws[SW], wd[SW], wu[SW], wv[SW];
    R s0[SW], s1[SW], s2[SW];
    double se[SW];
    R rc[2][RC];           // the segment's row constants: 1 / (dx cfl/2) of its east-west edges, dt / area
};

constexpr int strip_min_ctas(int mode, bool eddy, int real_bytes)
{
    return (eddy || (real_bytes == 8 && mode != MODE_STAGE2)) ? 4 : 5;
}

template <typename R, int MODE, bool SPH, bool COR, int FRIC, bool EDDY>
__global__ void __launch_bounds__(SW, strip_min_ctas(MODE, EDDY, (int)sizeof(R))) rk2_strip_kernel(const Rk2Args<R> a,
                                                                                                    int SH)
{
    constexpr bool UPDATE = (MODE == MODE_STAGE1 || MODE == MODE_STAGE2);
    __shared__ Strip<R> sm;
    after_previous();
    const int lane = threadIdx.x, l = lane + 1;
    const int nx = a.nx, ny = a.ny;
    const int strips_x = (nx + SO - 1) / SO;
    const int sx = blockIdx.x % strips_x, sy = blockIdx.x / strips_x;
    const int ra = sy * SH;
    const int rb = min(ra + SH, ny);
    const int i = sx * SO - 2 + lane;
    const bool col_valid = (i >= 0 && i < nx);
    const bool col_edge = (i >= 1 && i < nx);                      // edges exist in column i
    const bool out_lane = (lane >= 2 && lane <= SW - 3 && i < nx);
    const bool ew_edge = col_edge && lane >= 2 && lane <= SW - 2;  // west edges this strip needs
    const bool ew_grad = (i > 0 && i < nx - 1);

    R dt = R(0);
    if (UPDATE) dt = stage_dt<R>(a);
    const R inv2 = R(1) / (a.m.dyl[0] * a.half_cfl);
    const R dyl = col_valid ? a.m.dyl[i] : R(1);
    R speed = R(0);        // largest wave speed of the column's north-south edges
    double cfl = 0.0;      // largest 1/dt of its east-west edges
    int negfix = 0;
    // The row constants of the segment's rows, one division each by the
    // strip's threads instead of one per cell (the same expressions; read
    // after the loop's first barrier).
    const bool rc_sm = (rb - ra) <= RC;
    if (rc_sm)
        for (int t = lane; t < rb - ra; t += SW) {
            const int rr = ra + t;
            sm.rc[0][t] = R(1) / (a.m.dxb[rr] * a.half_cfl);
            if (UPDATE) sm.rc[1][t] = dt / a.m.area[rr];
        }

    auto load = [&](int r) {
        Raw<R> x;
        x.s = x.uh = x.vh = x.e = R(0);
        if (col_valid && r >= 0 && r < ny) {
            const int64_t row = (int64_t)r * a.P;
            x.s = (a.stg + row)[i]; x.uh = (a.uh + row)[i]; x.vh = (a.vh + row)[i]; x.e = (a.elv + row)[i];
        }
        return x;
    };
    Raw<R> nxt = load(ra - 2);
    // ring slots of rows r, r-1, r-2, rotated each row
    int t0 = (ra + 1) % 3, t1 = (t0 + 2) % 3, t2 = (t0 + 1) % 3;
    for (int r = ra - 2, k = 0; r <= rb + 1; r++, k++, t2 = t1, t1 = t0, t0 = (t0 == 2) ? 0 : t0 + 1) {
        __syncthreads();   // every thread is done with the entries this row rewrites
        const Raw<R> cur = nxt;
        if (r + 1 <= rb + 1) nxt = load(r + 1);
        if (UPDATE && out_lane && r + 1 >= ra && r + 1 < rb) {
            const int64_t o = (int64_t)(r + 1) * a.P + i;
            if (FRIC != FRIC_NONE) prefetch_l2(a.nsq + o);
            if (MODE == MODE_STAGE2) {
                prefetch_l2(a.stg0 + o);
                prefetch_l2(a.uh0 + o);
                prefetch_l2(a.vh0 + o);
                if (a.max_stage) prefetch_l2(a.max_stage + o);
            }
        }
        bool fixed;
        const Cell<R> cC = fix_up<R>(cur, col_valid && r >= 0 && r < ny, fixed);
        if (UPDATE && fixed && out_lane && r >= ra && r < rb) negfix++;
        sm.stg[t0][l] = cC.stg; sm.dep[t0][l] = cC.dep; sm.u[t0][l] = cC.u; sm.v[t0][l] = cC.v; sm.elv[t0][l] = cC.elv;

        // (the column's own rows come back from shared memory: kept in registers
        // they cost the fifth CTA)
        Cell<R> cA, cB;        // rows r-2, r-1
        {
            cA.stg = sm.stg[t2][l]; cA.dep = sm.dep[t2][l]; cA.u = sm.u[t2][l]; cA.v = sm.v[t2][l]; cA.elv = sm.elv[t2][l];
            cB.stg = sm.stg[t1][l]; cB.dep = sm.dep[t1][l]; cB.u = sm.u[t1][l]; cB.v = sm.v[t1][l]; cB.elv = sm.elv[t1][l];
        }
        EdgeRes<R> e_n, e_w;   // the north edge and the west edge of row r-2
        e_n.f[0] = e_n.f[1] = e_n.f[2] = R(0);
        e_n.es_pos = e_n.es_neg = 0.0;
        e_w = e_n;
        if (k >= 2) {
            // North-south gradient of row r-1, its faces, and the edge below it.
            const int e = r - 1;
            Grad<R> g;
            g.ds = g.dd = g.du = g.dv = R(0);
            if (col_valid && e > 0 && e < ny - 1) g = limited<R>(cA, cB, cC, a.theta);
            if (k >= 3 && col_edge && e >= 1 && e <= ny - 1) {
                EddyIn<R> eddy;
                if (EDDY) {
                    eddy.ev_n = a.ev[(int64_t)(e - 1) * a.P + i];
                    eddy.ev_p = a.ev[(int64_t)e * a.P + i];
                    eddy.du = cB.u - cA.u; eddy.dv = cB.v - cA.v; eddy.vel_div = dyl;
                }
                R ms;
                Face<R> north;
                north.s = sm.ns[lane]; north.d = sm.nd[lane]; north.u = sm.nu[lane]; north.v = sm.nv[lane];
                edge_faces<R, true, EDDY>(north, cA.dep, cA.elv, face_below(cB, g), cB.dep, cB.elv, a.m.dxb[e], e_n,
                                          ms, a.flux_variant, eddy);
                if (MODE != MODE_STAGE2) speed = rmax(speed, ms);   // stage 2 writes no CFL
                // the boundary-flux lines (rows n_ext and ny - n_ext): tested
                // on the row first, the same for the whole strip
                if (MODE != MODE_CFL && (e == ny - a.n_ext || e == a.n_ext) && a.lines && i >= a.n_ext &&
                    i <= nx - a.n_ext - 1) {
                    if (e == ny - a.n_ext) a.lines[i] = (double)e_n.f[0];
                    if (e == a.n_ext) a.lines[nx + ny + i] = (double)e_n.f[0];
                }
            }
            const Face<R> north = face_above(cB, g);
            sm.ns[lane] = north.s; sm.nd[lane] = north.d; sm.nu[lane] = north.u; sm.nv[lane] = north.v;
        }
        const int q = r - 2;   // the row being updated
        if (k >= 4) {
            // Its west edges, from the east faces of the columns to the west.
            if (ew_edge && q >= 1 && q <= ny - 1) {
                const R inv1 = rc_sm ? sm.rc[0][q - ra] : R(1) / (a.m.dxb[q] * a.half_cfl);
                const int fb = r & 1;
                Face<R> n;
                n.s = sm.fs[fb][l - 1]; n.d = sm.fd[fb][l - 1]; n.u = sm.fu[fb][l - 1]; n.v = sm.fv[fb][l - 1];
                Face<R> west;
                west.s = sm.ws[lane]; west.d = sm.wd[lane]; west.u = sm.wu[lane]; west.v = sm.wv[lane];
                EddyIn<R> eddy;
                if (EDDY) {
                    const int64_t oe = (int64_t)q * a.P + i;
                    eddy.ev_n = a.ev[oe - 1]; eddy.ev_p = a.ev[oe];
                    eddy.du = cA.u - sm.u[t2][l - 1]; eddy.dv = cA.v - sm.v[t2][l - 1];
                    eddy.vel_div = R(0.5) * (a.m.dxb[q] + a.m.dxb[q + 1]);
                }
                R ms;
                edge_faces<R, false, EDDY>(n, sm.dep[t2][l - 1], sm.elv[t2][l - 1], west, cA.dep, cA.elv, dyl, e_w, ms,
                                           a.flux_variant, eddy);
                if (MODE != MODE_STAGE2) cfl = rmax(cfl, cfl_rate<R>(ms, inv1));
                if (MODE != MODE_CFL && (i == nx - a.n_ext || i == a.n_ext) && a.lines && q >= a.n_ext &&
                    q <= ny - a.n_ext - 1) {
                    if (i == nx - a.n_ext) a.lines[nx + q] = (double)e_w.f[0];
                    if (i == a.n_ext) a.lines[2 * nx + ny + q] = (double)e_w.f[0];
                }
            }
            if (MODE != MODE_CFL) { sm.f0[l] = e_w.f[0]; sm.f1[l] = e_w.f[1]; sm.f2[l] = e_w.f[2]; sm.es[l] = e_w.es_neg; }
        }
        // What stage 2's update reads, on its way before the gradient and the
        // barrier that precede it: stage 2 267 -> 254 us at 2048^2 FP64, 220 ->
        // 207 FP32 (the other modes read less and spill with it: midpoint
        // 144.5 -> 146.5 us a step at 930^2).
        R Um_uh = R(0), Um_vh = R(0), nsq = R(0);
        Stage2Reg<R> in;
        in.s_ = in.uh_ = in.vh_ = in.mx_ = R(0);
        if (MODE == MODE_STAGE2 && k >= 4 && out_lane) {
            const int64_t o = (int64_t)q * a.P + i;
            Um_uh = a.uh[o]; Um_vh = a.vh[o];
            in.s_ = a.stg0[o]; in.uh_ = a.uh0[o]; in.vh_ = a.vh0[o];
            if (a.max_stage) in.mx_ = a.max_stage[o];
            if (FRIC != FRIC_NONE) nsq = a.nsq[o];
        }
        if (k >= 3 && r <= rb) {
            // East-west gradient of row r-1 (its neighbours' values were
            // written before this row's barrier) and its two faces, for the
            // west edges in the next row's pass.
            Grad<R> g;
            g.ds = g.dd = g.du = g.dv = R(0);
            if (ew_grad) {
                Cell<R> lo, hi;
                lo.stg = sm.stg[t1][l - 1]; lo.dep = sm.dep[t1][l - 1]; lo.u = sm.u[t1][l - 1]; lo.v = sm.v[t1][l - 1];
                hi.stg = sm.stg[t1][l + 1]; hi.dep = sm.dep[t1][l + 1]; hi.u = sm.u[t1][l + 1]; hi.v = sm.v[t1][l + 1];
                g = limited<R>(lo, cB, hi, a.theta);
            }
            const Face<R> east = face_above(cB, g);
            const int fb = (r + 1) & 1;
            sm.fs[fb][l] = east.s; sm.fd[fb][l] = east.d; sm.fu[fb][l] = east.u; sm.fv[fb][l] = east.v;
            const Face<R> west = face_below(cB, g);
            sm.ws[lane] = west.s; sm.wd[lane] = west.d; sm.wu[lane] = west.u; sm.wv[lane] = west.v;
        }
        if (MODE != MODE_CFL && k >= 4) {
            __syncthreads();
            if (out_lane) {
                EdgeRes<R> e_s, e_e;
                cA.stg = sm.stg[t2][l]; cA.dep = sm.dep[t2][l]; cA.u = sm.u[t2][l]; cA.v = sm.v[t2][l]; cA.elv = sm.elv[t2][l];
                e_s.f[0] = sm.s0[lane]; e_s.f[1] = sm.s1[lane]; e_s.f[2] = sm.s2[lane];
                e_s.es_pos = sm.se[lane]; e_s.es_neg = 0.0;
                e_e.f[0] = sm.f0[l + 1]; e_e.f[1] = sm.f1[l + 1]; e_e.f[2] = sm.f2[l + 1];
                e_e.es_neg = sm.es[l + 1];
                e_e.es_pos = 0.0;
                const int64_t o = (int64_t)q * a.P + i;
                if (MODE == MODE_STAGE2) {
                    if (!(cA.dep > K<R>::min_depth())) Um_uh = Um_vh = R(0);
                } else if (UPDATE || SPH) {
                    fixed_momenta<R>(a, o, cA, Um_uh, Um_vh);
                }
                const CellFlux<R> f = cell_flux<R, SPH, COR>(a, i, q, cA, Um_uh, Um_vh, e_s, e_n, e_w, e_e);
                if (MODE == MODE_FLUX) {
                    // the cell's dt-independent update terms, for the stage-1 update once dt is known
                    a.cs.d[0][o] = f.d[0]; a.cs.d[1][o] = f.d[1]; a.cs.d[2][o] = f.d[2];
                    a.cs.eu[o] = f.eu; a.cs.ev[o] = f.ev;
                } else {
                    fv_apply<R, MODE>(a, i, q, cA, Um_uh, Um_vh, f, rc_sm ? sm.rc[1][q - ra] : dt / a.m.area[q],
                                      [&] {
                                          const R n = MODE == MODE_STAGE2 ? nsq : FRIC == FRIC_NONE ? R(0) : a.nsq[o];
                                          return friction_factor<R, FRIC>(a, n, cA, dt);
                                      },
                                      in);
                }
            }
        }
        sm.s0[lane] = e_n.f[0]; sm.s1[lane] = e_n.f[1]; sm.s2[lane] = e_n.f[2]; sm.se[lane] = e_n.es_pos;
    }

    if (MODE != MODE_STAGE2 && (a.write_cfl || MODE == MODE_CFL || MODE == MODE_FLUX)) {
        cfl = rmax(cfl, cfl_rate<R>(speed, inv2));   // (the product with 1/dx rises with the speed)
        for (int o = 16; o > 0; o >>= 1) cfl = fmax(cfl, __shfl_down_sync(FULL, cfl, o));
        if ((lane & 31) == 0 && cfl > 0.0)
            atomicMax(&a.sc->max_dt_inv_bits, (unsigned long long)__double_as_longlong(cfl));
    }
    if (UPDATE) {
        negfix = __reduce_add_sync(FULL, negfix);
        if ((lane & 31) == 0 && negfix)
            atomicAdd((unsigned long long *)&a.sc->negative_depth_fix_counter, (unsigned long long)negfix);
    }
}

// CTAs of a launch with sh rows per strip segment.
int64_t fv_ctas(int nx, int ny, int sh) { return (int64_t)((nx + SO - 1) / SO) * ((ny + sh - 1) / sh); }

// Rows per strip segment for a grid (SWALS_FV_ROWS sets it): the count with
// the least estimate, over the rounds in which an SM takes its `resident`
// CTAs, of
//   (rows + 1.5) x sum of (2, or 0.75 after the first round, + CTAs of the round).
// The 1.5 rows stand for the lead-in, whose rows do part of a row's work; the
// 2 for the chain of a row, that few CTAs leave bare and that the CTAs of a
// later round mostly start under.  `resident` is the kernel's own: a round of
// four is full where one of five would not be.  Measured on the B200, us a
// launch, the estimate's rows (best of 1 .. 32): flux kernel FP64 300 x 200 2
// 15.2, 600 x 500 6 28.5, 930^2 13 57.8, 1275 x 879 6 72.6 (10: 72.5), 2048^2
// 20 209.5 (16: 207.6), FP32 1531 x 1021 7 73.7 (9: 72.1); stage 2 1 16.7, 6
// 33.1, 13 70.4 (5: 69.9), 7 86.7, 16 252.9, 7 90.5 (9: 88.4); midpoint's two
// stages 930^2 13 137.0, 500 x 700 6 74.2: 0.5 % above the best on average, 2.4
// at most.  One line for all kernels over fewer counts had taken 145.1 and
// 80.0 for the last two, 79.9 for the flux kernel at 1275 x 879.
int fv_rows(int nx, int ny, int resident)
{
    const char *e = getenv("SWALS_FV_ROWS");
    if (e && atoi(e) > 0) return atoi(e);
    static int sms = 0;
    if (sms == 0) {
        int dev = 0, n = 148;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms = n;
    }
    int best = 0;
    double best_cost = 0.0;
    for (int sh = 1; sh <= 32; sh++) {
        double t = 0.0, chain = 2.0;
        for (double left = (double)fv_ctas(nx, ny, sh) / sms; left > 1e-9; left -= resident, chain = 0.75)
            t += chain + std::min(std::ceil(left), (double)resident);
        const double cost = (sh + 1.5) * t;
        if (best == 0 || cost < best_cost) {
            best = sh;
            best_cost = cost;
        }
    }
    return best;
}

}  // namespace

template <typename R, int MODE, bool SPH, bool COR, int FRIC>
cudaError_t launch_stage_stream(const Rk2Args<R> &a, cudaStream_t s)
{
    // Stage 2 takes the first stage's dt and accumulates no CFL maximum: its
    // kernels leave the edges' wave-speed candidates out.
    if (MODE == MODE_STAGE2 && a.write_cfl) return cudaErrorInvalidValue;
    const bool eddy = MODE != MODE_CFL && (a.flux_variant & FLUX_EDDY);
    const int SH = fv_rows(a.nx, a.ny, strip_min_ctas(MODE, eddy, (int)sizeof(R)));
    const int blocks = (int)fv_ctas(a.nx, a.ny, SH);
    if constexpr (MODE != MODE_CFL) {
        if (eddy) {
            return launch_behind(rk2_strip_kernel<R, MODE, SPH, COR, FRIC, true>, blocks, SW, 0, s, a, SH);
        }
    }
    return launch_behind(rk2_strip_kernel<R, MODE, SPH, COR, FRIC, false>, blocks, SW, 0, s, a, SH);
}

#define SWALS_INST(R, MODE, SPH, COR, FRIC) \
    template cudaError_t launch_stage_stream<R, MODE, SPH, COR, FRIC>(const fv::Rk2Args<R> &, cudaStream_t);
#define SWALS_INST_F(R, MODE, SPH, COR) \
    SWALS_INST(R, MODE, SPH, COR, fv::FRIC_MANNING) SWALS_INST(R, MODE, SPH, COR, fv::FRIC_CHEZY) \
    SWALS_INST(R, MODE, SPH, COR, fv::FRIC_NONE)
#define SWALS_INST_M(R, SPH, COR) \
    SWALS_INST_F(R, fv::MODE_CFL, SPH, COR) SWALS_INST_F(R, fv::MODE_STAGE1, SPH, COR) \
    SWALS_INST_F(R, fv::MODE_FLUX, SPH, COR) \
    SWALS_INST_F(R, fv::MODE_STAGE2, SPH, COR)
SWALS_INST_M(double, false, false)
SWALS_INST_M(double, true, false)
SWALS_INST_M(double, true, true)
SWALS_INST_M(float, false, false)
SWALS_INST_M(float, true, false)
SWALS_INST_M(float, true, true)

}  // namespace swals
