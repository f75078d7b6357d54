// linear_pair.cu -- two linear leapfrog steps in one pass over the grid.
//
// The single-step kernels (linear.cu) move 9 planes per step and run at 0.87 -
// 0.96 of the HBM bandwidth; on grids beyond L2 only fewer passes make a step
// cheaper.  This kernel reads the state once, applies
// domain_mod_linear_solver_include.f90:58-571 twice and writes it once: 9
// planes for two steps (11 with the friction work of
// leapfrog_linear_plus_nonlinear_friction).  On grids in L2 it halves the
// launches instead.
//
// A CTA is one warp: SMs fill evenly and its row segments can be short.  It
// owns a strip of 30 lanes x 16 bytes (60 FP64 or 120 FP32 columns) plus one
// lane of halo either side -- two steps reach two columns, and a lane holds at
// least two -- and marches down a segment of rows plus two at each end.  When
// row r arrives (by 16-byte cp.async, two rows ahead, in a ring that also
// keeps row r-1):
//   stage of step 1 in row r, momenta of step 1 in row r-1,
//   stage of step 2 in row r-1, momenta of step 2 in row r-2, row r-2 out.
// What a row needs of the results before stays in registers, neighbouring
// columns come by shuffle, and there is no barrier in the march.  The warp
// issues more instructions than it waits for memory, so what two rows or both
// steps share is formed once: VH x edge length and the two-point averages of a
// row serve the next row too, g dt/area x face depth and the Coriolis factor
// of a wet face (truly linear solver) both steps, the row constants (dt / area
// and so on) the whole strip; a segment away from the sides selects nothing.
// 112 -> 93 thread instructions a cell and step, 3600 x 2400 FP32
// Coriolis 43.7 -> 36.3 us a step.  Products and sums keep the single step's
// operands and order, so the results are the same bits.
//
// 16-byte lanes start on 16-byte boundaries (strips every 480 bytes, 15 whole
// sectors); planes that linear_pair_fits refuses step one at a time.  8-byte
// lanes with twice the warps are no faster (FP32 38.3).
//
// Measured on the B200, us a step, one step at a time / in pairs: 4096^2 FP64
// 212 / 113, 8192^2 787 / 427 (a pair moves 72 B a cell: 5.3 and 5.7 TB/s,
// 0.83 and 0.88 of the copy bandwidth), FP32 111 / 62, 3600 x 2400 FP32
// Coriolis 71.6 / 36.3, 1200 x 800 Coriolis 20.5 / 10.5, 400^2 with 9 gauges
// 9.4 / 4.9, 200 x 150 7.2 / 3.3; with Manning friction 1501 x 1001 Coriolis
// 58.0 / 28.2, 3000 x 2000 FP32 114 / 45.7.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "pair_common.cuh"

namespace swals {
namespace {

using pair::FULL;
using pair::cp16;

constexpr int SLOTS = 4;    // ring slots per warp: rows r - 1, r and two in flight
constexpr int GROUP = 16;   // instances of a batch whose CTAs are neighbours

// Warps per SM that the register cap leaves room for (168 a thread for 12).
// Fewer do not hide the latencies, more spill: 3600 x 2400 FP32 Coriolis 37.3
// us a step at 12, 69 at 16 (240 bytes of spills).  With the friction work the
// two steps' square roots and quotients bind, and FP64 takes 207 registers:
// 1501 x 1001 Coriolis 29.3 us a step at 8, 52.3 with spills at 16.
constexpr int pair_warps(bool nlf, int real_bytes) { return nlf && real_bytes == 8 ? 8 : 12; }

// Row constants of a segment, rows ra - 2 .. (clamped to the grid): dt/area,
// distance_bottom_edge(r + 1), g dt/area, g dt/mean area, dt cor/2 at the row
// and at its north edge.
template <typename R> struct __align__(16) RowConst {
    R cs, dxb1, cu, cv, dtc, dtj;
};

template <typename R, bool COR, bool TL, bool NLF, bool GAUGES>
__global__ void __launch_bounds__(32, pair_warps(NLF, (int)sizeof(R))) linear_pair_kernel(const LinearPair<R> a, int SH, int nstrips)
{
    constexpr int CPL = 16 / (int)sizeof(R);
    constexpr int OUTC = 30 * CPL;
    constexpr int NP = NLF ? 7 : 5;      // UH, VH, STG, ELV, max_stage and friction work at UH, VH of row r-1
    constexpr bool AVG = COR || NLF;     // the two-point averages of the other momentum
    typedef typename pair::Vec<R>::T V;
    struct Face { R gu[CPL], gv[CPL], cu[CPL], cv[CPL], wi[CPL], wj[CPL]; };
    extern __shared__ __align__(16) unsigned char pair_smem[];
    RowConst<R> *rc = reinterpret_cast<RowConst<R> *>(pair_smem + sizeof(V) * 32 * NP * SLOTS);
    const int lane = threadIdx.x;
    V *ring = reinterpret_cast<V *>(pair_smem);   // [slot][plane][lane]

    const int nx = a.p.nx, ny = a.p.ny;
    const int64_t P = a.p.pitch;
    // Instances in groups of GROUP: a group's CTAs on the same rows and columns
    // are neighbours and share ELV in L2; groups follow one another (256
    // instances of 3600 x 2400 FP32 8.52 ms a step in one group, 8.37 in groups).
    const int tiles = nstrips * ((ny + SH - 1) / SH);
    const int group = min(GROUP, a.nbatch);
    const int b0 = (int)(blockIdx.x / ((unsigned)group * tiles)) * group;
    const int in_group = (int)(blockIdx.x - (unsigned)b0 * tiles), members = min(group, a.nbatch - b0);
    const int b = b0 + in_group % members;
    const int tile = in_group / members;
    const int strip = tile % nstrips;
    const int ra = (tile / nstrips) * SH;
    const int rb = min(ra + SH, ny);
    const R half = K<R>::half(), zero = K<R>::zero(), one = K<R>::one(), mad = K<R>::min_depth();
    const R dt = a.dt, msl = a.msl;

    for (int k = lane; k < rb - ra + 4; k += 32) {
        const int r = min(max(ra - 2 + k, 0), ny - 1);
        const R g = K<R>::gravity();
        RowConst<R> c;
        c.cs = dt / a.m.area[r];
        c.cu = g * dt / a.m.area[r];
        c.cv = g * dt / (half * (a.m.area[r] + a.m.area[min(r + 1, ny - 1)]));
        c.dxb1 = a.m.dxb[r + 1];
        c.dtc = COR ? dt * a.m.cor[r] * half : zero;
        c.dtj = COR ? dt * a.m.cor_be[r + 1] * half : zero;
        rc[k] = c;
    }
    pair::GaugeRows gauges(reinterpret_cast<int *>(rc + (SH + 4)), a.g_sites, GAUGES ? a.g_n : 0, ny, ra - 2, rb - ra + 4,
                           lane);
    __syncthreads();
    if (GAUGES) gauges.ready(rb - ra + 4, lane);
    after_previous();   // (the metrics and gauge sites above are no kernel's output)
    let_next_start();
    const int rec = GAUGES ? (a.g_count ? *a.g_count : 0) : 0;

    const int64_t io = (int64_t)b * a.inst_stride;
    const R *pl[4] = {a.p.uh + io, a.p.vh + io, a.p.stg + io, a.p.elv};
    R *stg_o = a.p.stg_o + io, *uh_o = a.p.uh_o + io, *vh_o = a.p.vh_o + io;
    R *max_stage = a.p.max_stage ? a.p.max_stage + (int64_t)b * a.max_stride : nullptr;
    const int c0 = strip * OUTC + (lane - 1) * CPL;          // this lane's first column
    const bool out = lane >= 1 && lane <= 30 && c0 < nx;
    const int src = c0 < 0 ? 0 : min(max(nx - c0, 0), CPL) * (int)sizeof(R);
    const int cl = src ? c0 : 0;                             // an address inside the row for zero-filled lanes
    const bool whole = c0 + CPL <= nx;
    const bool first = c0 == 0;                              // UH west of column 0 is column 0's
    R dyl[CPL + 1];
    unsigned st_m = 0u, mo_m = 0u, ms_m = 0u;                // the columns against xL .. xU
#pragma unroll
    for (int c = 0; c <= CPL; c++) dyl[c] = a.m.dyl[min(max(c0 + c, 0), nx)];
#pragma unroll
    for (int c = 0; c < CPL; c++) {
        const int col = c0 + c;
        st_m |= (unsigned)(col >= a.xl + 1 && col <= a.xu - 1) << c;
        mo_m |= (unsigned)(col >= a.xl && col <= a.xu - 1) << c;
        ms_m |= (unsigned)(col >= a.xl && col <= a.xu) << c;
    }
    // the gauges in the warp's output columns
    auto record = [&](int step, int row, const R(&s)[CPL], const R(&u)[CPL], const R(&v)[CPL]) {
        if (rec + step >= a.g_capacity) return;
        gauges.on_row(row - (ra - 2), strip * OUTC, strip * OUTC + OUTC - 1, lane, [&](unsigned, bool hit, int col, int q) {
            // the lane with the site fetches the values of its cell
            const int from = 1 + col / CPL, comp = col % CPL;
            auto fetch = [&](const R(&x)[CPL]) {
                R y = __shfl_sync(FULL, x[0], from);
#pragma unroll
                for (int c = 1; c < CPL; c++) {
                    const R z = __shfl_sync(FULL, x[c], from);
                    if (comp == c) y = z;
                }
                return (double)y;
            };
            double *d = a.g_rec + (((int64_t)(rec + step) * a.nbatch + b) * a.g_n + q) * a.g_vals;
            const double fs = fetch(s);
            if (hit) d[0] = fs;
            if (a.g_vals == 3) {
                const double fu = fetch(u), fv = fetch(v);
                if (hit) { d[1] = fu; d[2] = fv; }
            }
        });
    };
    // the lane's component on the west and east boundary-flux lines, or -1
    const int ln_e = (a.lines && out) ? nx - a.n_ext - 1 - c0 : -1, ln_w = (a.lines && out) ? a.n_ext - 1 - c0 : -1;

    const int r0 = max(ra - 2, 0);
    auto issue = [&](int r, int slot) {
        if (r <= rb + 1) {
            V *s = ring + (size_t)slot * NP * 32 + lane;
            const int rr = min(r, ny - 1);
            const int64_t o = (int64_t)rr * P + cl;
            const int n = r < ny ? src : 0;
#pragma unroll
            for (int k = 0; k < 4; k++) cp16(s + k * 32, pl[k] + o, n);
            // max_stage and the friction work of the row before
            const bool mx = max_stage && r - 1 >= ra && r - 1 < rb && out;
            cp16(s + 4 * 32, mx ? max_stage + (int64_t)(r - 1) * P + cl : pl[2] + o, mx ? src : 0);
            if (NLF) {
                const int64_t of = (int64_t)min(max(r - 1, 0), ny - 1) * P + cl;
                cp16(s + 5 * 32, a.fw + of, src);
                cp16(s + 6 * 32, a.fw + a.fw_plane + of, src);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    auto get = [&](const V *s, int k, R(&v)[CPL]) {
        const V x = s[k * 32];
        const R *xs = reinterpret_cast<const R *>(&x);
#pragma unroll
        for (int c = 0; c < CPL; c++) v[c] = xs[c];
    };
    auto west = [&](const R(&v)[CPL], R(&o)[CPL]) {
        const R up = __shfl_up_sync(FULL, v[CPL - 1], 1);
        o[0] = first ? v[0] : up;
#pragma unroll
        for (int c = 1; c < CPL; c++) o[c] = v[c - 1];
    };
    auto east = [&](const R(&v)[CPL], R(&o)[CPL]) {
        const R dn = __shfl_down_sync(FULL, v[0], 1);
#pragma unroll
        for (int c = 0; c + 1 < CPL; c++) o[c] = v[c + 1];
        o[CPL - 1] = dn;
    };
    // One segment.  INNER: every column of the strip and every row of the
    // march is in xL+1 .. xU-1, yL+1 .. yU-1, so nothing is selected.
    auto march = [&](auto inner) {
        constexpr bool INNER = decltype(inner)::value;
        // New stage of row r (:92-115); vd, vds: VH x distance_bottom_edge
        // at the row's north and south edges.
        auto stage = [&](int r, const RowConst<R> &k, const R(&s)[CPL], const R(&u)[CPL], const R(&uw)[CPL],
                         const R(&vd)[CPL], const R(&vds)[CPL], R(&o)[CPL]) {
            const bool row = r >= a.yl + 1 && r <= a.yu - 1;
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                const R t1 = (u[c] - uw[c]) * dyl[c];
                const R t2 = vd[c] - vds[c];
                const R n = s[c] - k.cs * (t1 + t2);
                o[c] = (INNER || (row && ((st_m >> c) & 1u))) ? n : s[c];
            }
        };
        // Face depths (:353-370; not truly linear: of the new stage) times
        // g dt/area, and the Coriolis factor where the face is wet.  (Half of
        // a wet face's sum is exact, so the fma rounds as the difference does.)
        auto faces = [&](const RowConst<R> &k, const R(&e)[CPL], const R(&ee)[CPL], const R(&en)[CPL], const R(&s)[CPL],
                         const R(&se)[CPL], const R(&sn)[CPL], Face &f) {
            const R lim = -mad + msl;
            const R dtc0 = k.dtc * zero, dtj0 = k.dtj * zero;
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                R hi, hj;
                if (TL) {
                    const bool w0 = e[c] < lim;
                    hi = (w0 && ee[c] < lim) ? fma(-half, ee[c] + e[c], msl) : zero;
                    hj = (en[c] < lim && w0) ? fma(-half, en[c] + e[c], msl) : zero;
                } else {
                    const bool w0 = s[c] - e[c] > mad;
                    hi = (w0 && se[c] - ee[c] > mad) ? (half * ((se[c] + s[c]) - (ee[c] + e[c]))) : zero;
                    hj = (sn[c] - en[c] > mad && w0) ? (half * ((sn[c] + s[c]) - (en[c] + e[c]))) : zero;
                    f.wi[c] = (hi > zero) ? one : zero;
                    f.wj[c] = (hj > zero) ? one : zero;
                }
                f.gu[c] = k.cu * hi;
                f.gv[c] = k.cv * hj;
                if (COR) {
                    f.cu[c] = (hi > zero) ? k.dtc : dtc0;
                    f.cv[c] = (hj > zero) ? k.dtj : dtj0;
                }
            }
        };
        // Momenta of row j (:225-567) from the old momenta u, v, their
        // two-point averages hvs (VH of row j-1 and its east neighbour),
        // hu, hun (UH of rows j, j+1 and its west neighbour) and the new
        // stage s, se, sn; hv: the average of this row, for the next.
        auto momenta = [&](int j, R dxb1, const R(&u)[CPL], const R(&v)[CPL], const R(&s)[CPL], const R(&se)[CPL],
                           const R(&sn)[CPL], const Face &k, const R(&hvs)[CPL], const R(&hu)[CPL], const R(&hun)[CPL],
                           const R(&fu)[CPL], const R(&fv)[CPL], R(&ou)[CPL], R(&ov)[CPL], R(&hv)[CPL]) {
            const bool row = j >= a.yl && j <= a.yu - 1;
            if (AVG) {
                R ve[CPL];
                east(v, ve);
#pragma unroll
                for (int c = 0; c < CPL; c++) hv[c] = half * (v[c] + ve[c]);
            }
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                R uu = u[c], vv = v[c];
                if (!TL) {   // wet factors
                    uu = uu * k.wi[c];
                    vv = vv * k.wj[c];
                }
                uu = uu - k.gu[c] * (se[c] - s[c]) * dyl[c + 1];
                vv = vv - k.gv[c] * (sn[c] - s[c]) * dxb1;
                if (AVG) {
                    const R v4 = (!INNER && j == 0 ? hv[c] : hvs[c]) + hv[c];
                    const R u4 = hu[c] + hun[c];
                    if (COR) {
                        uu = uu + k.cu[c] * v4;
                        vv = vv - k.cv[c] * u4;
                    }
                    if (NLF) {
                        uu = friction_multiplier_line(one + a.lin_fric_dt, dt, fu[c], u[c], half * v4) * uu;
                        vv = friction_multiplier_line(one + a.lin_fric_dt, dt, fv[c], v[c], half * u4) * vv;
                    }
                }
                if (!NLF && a.lin_fric) {
                    uu = a.lin_fric_mult * uu;
                    vv = a.lin_fric_mult * vv;
                }
                const bool ok = INNER || (row && ((mo_m >> c) & 1u));
                ou[c] = ok ? uu : u[c];
                ov[c] = ok ? vv : v[c];
            }
        };

        // Of row r-1: stage of step 1, VH x edge, average of UH; of row
        // r-2: average of VH; max_stage with the stage of step 1, momenta
        // of step 1, stage of step 2, VH x edge, average of UH, faces; of
        // row r-3: average of step 1's VH.
        R a1[CPL], vd1[CPL], hu1[CPL], hv2[CPL], f2[CPL], g2[CPL];
        R m2[CPL], uA2[CPL], vA2[CPL], b2[CPL], vdA2[CPL], huA2[CPL], hvA3[CPL], e2[CPL];
        Face k2f;
#pragma unroll
        for (int c = 0; c < CPL; c++) {
            a1[c] = vd1[c] = hu1[c] = hv2[c] = f2[c] = g2[c] = zero;
            m2[c] = uA2[c] = vA2[c] = b2[c] = vdA2[c] = huA2[c] = hvA3[c] = e2[c] = zero;
            k2f.gu[c] = k2f.gv[c] = k2f.cu[c] = k2f.cv[c] = k2f.wi[c] = k2f.wj[c] = zero;
        }
        auto step = [&](int r, int slot) {
            issue(r + 2, (slot + 2) % SLOTS);   // (into the slot of row r-2)
            asm volatile("cp.async.wait_group 2;\n" ::);
            const V *s = ring + (size_t)slot * NP * 32 + lane;
            const V *s1 = ring + (size_t)((slot + SLOTS - 1) % SLOTS) * NP * 32 + lane;
            R u[CPL], v[CPL], st[CPL], e[CPL], u1[CPL], v1[CPL], e1[CPL], f1[CPL], g1[CPL];
            get(s, 0, u); get(s, 1, v); get(s, 2, st); get(s, 3, e);
            get(s1, 0, u1); get(s1, 1, v1); get(s1, 3, e1);
#pragma unroll
            for (int c = 0; c < CPL; c++) f1[c] = g1[c] = zero;
            if (NLF) { get(s, 5, f1); get(s, 6, g1); }
            const RowConst<R> &k0 = rc[r - (ra - 2)];
            const RowConst<R> &k1 = rc[max(r - 1 - (ra - 2), 0)];
            const RowConst<R> &k2 = rc[max(r - 2 - (ra - 2), 0)];

            // step 1: stage of row r, momenta of row r-1
            R uw[CPL], vd[CPL], hu[CPL], hv[CPL], sA[CPL], ae[CPL], ee[CPL], uA[CPL], vA[CPL];
            Face k1f;
            west(u, uw);
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                vd[c] = v[c] * k0.dxb1;
                hu[c] = AVG ? half * (u[c] + uw[c]) : zero;
                hv[c] = zero;
            }
            stage(r, k0, st, u, uw, vd, vd1, sA);
            east(a1, ae);
            east(e1, ee);
            faces(k1, e1, ee, e, a1, ae, sA, k1f);
            momenta(r - 1, k1.dxb1, u1, v1, a1, ae, sA, k1f, hv2, hu1, hu, f1, g1, uA, vA, hv);
            if (a.lines && r - 1 >= ra && r - 1 < rb) {
                const int j = r - 1;
                if (out && (j == ny - a.n_ext - 1 || j == a.n_ext - 1)) {
#pragma unroll
                    for (int c = 0; c < CPL; c++)
                        if (c0 + c < nx) {
                            if (j == ny - a.n_ext - 1) a.lines[c0 + c] = vA[c];
                            if (j == a.n_ext - 1) a.lines[nx + ny + c0 + c] = vA[c];
                        }
                }
#pragma unroll
                for (int c = 0; c < CPL; c++) {
                    if (ln_e == c) a.lines[nx + j] = uA[c];
                    if (ln_w == c) a.lines[2 * nx + ny + j] = uA[c];
                }
            }

            // step 2: stage of row r-1, momenta of row r-2
            R uAw[CPL], vdA[CPL], huA[CPL], hvA[CPL], sB[CPL], be[CPL], uB[CPL], vB[CPL];
            west(uA, uAw);
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                vdA[c] = vA[c] * k1.dxb1;
                huA[c] = AVG ? half * (uA[c] + uAw[c]) : zero;
                hvA[c] = zero;
            }
            stage(r - 1, k1, a1, uA, uAw, vdA, vdA2, sB);
            east(b2, be);
            if (!TL) {
                R e2e[CPL];
                east(e2, e2e);
                faces(k2, e2, e2e, e1, b2, be, sB, k2f);
            }
            momenta(r - 2, k2.dxb1, uA2, vA2, b2, be, sB, k2f, hvA3, huA2, huA, f2, g2, uB, vB, hvA);

            // max_stage: row r-1 with step 1, row r-2 with step 2
            auto peak = [&](int row, const R(&x)[CPL], const R(&m)[CPL], R(&o)[CPL]) {
                const bool my = row >= a.yl && row <= a.yu;
#pragma unroll
                for (int c = 0; c < CPL; c++)
                    o[c] = ((INNER || (my && ((ms_m >> c) & 1u))) && x[c] > m[c]) ? x[c] : m[c];
            };
            R mx[CPL], m1[CPL];
            get(s, 4, mx);
            peak(r - 1, a1, mx, m1);
            const int q = r - 2;
            if (q >= ra && out) {   // (r <= rb + 1)
                const int64_t o = (int64_t)q * P + c0;
                R m[CPL];
                peak(q, b2, m2, m);
                if (INNER || whole) {
                    auto put = [&](R *p, const R(&x)[CPL]) {
                        V y;
                        R *ys = reinterpret_cast<R *>(&y);
#pragma unroll
                        for (int c = 0; c < CPL; c++) ys[c] = x[c];
                        *reinterpret_cast<V *>(p + o) = y;
                    };
                    put(stg_o, b2); put(uh_o, uB); put(vh_o, vB);
                    if (max_stage) put(max_stage, m);
                } else {
#pragma unroll
                    for (int c = 0; c < CPL; c++)
                        if (c0 + c < nx) {
                            stg_o[o + c] = b2[c]; uh_o[o + c] = uB[c]; vh_o[o + c] = vB[c];
                            if (max_stage) max_stage[o + c] = m[c];
                        }
                }
            }
            // gauges: step 1 on row r-1, step 2 on row r-2
            if (GAUGES && (gauges.on(r - 1 - (ra - 2)) || gauges.on(q - (ra - 2)))) {
                if (r - 1 >= ra && r - 1 < rb) record(0, r - 1, a1, uA, vA);
                if (q >= ra) record(1, q, b2, uB, vB);
            }
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                e2[c] = e1[c];
                vd1[c] = vd[c]; hu1[c] = hu[c]; hv2[c] = hv[c]; a1[c] = sA[c];
                uA2[c] = uA[c]; vA2[c] = vA[c]; vdA2[c] = vdA[c]; huA2[c] = huA[c]; hvA3[c] = hvA[c];
                b2[c] = sB[c]; m2[c] = m1[c];
                f2[c] = f1[c]; g2[c] = g1[c];
            }
            k2f = k1f;
        };
        // Row r0 reads u1, v1 and e1 of no row: zeros, as the carried values.
#pragma unroll
        for (int k = 0; k < 4; k++) ring[((SLOTS - 1) * NP + k) * 32 + lane] = V();
        issue(r0, 0);
        issue(r0 + 1, 1);
#pragma unroll 1
        for (int r = r0, slot = 0; r <= rb + 1; r++, slot = (slot + 1) % SLOTS) step(r, slot);
    };
    // Columns strip * OUTC - CPL .. (strip + 1) * OUTC + CPL - 1 and rows ra - 2 .. rb + 1.
    // (The friction form gains nothing from it: 31.1 against 29.6 us at 1501 x 1001.)
    if (!NLF && strip * OUTC - CPL >= a.xl + 1 && (strip + 1) * OUTC + CPL <= a.xu && ra - 2 >= a.yl + 1 && rb + 1 <= a.yu - 1)
        march(std::true_type());
    else
        march(std::false_type());
    asm volatile("cp.async.wait_group 0;\n" ::);

    if (GAUGES && a.g_count) {
        // Every CTA has read the record count before it counts itself done;
        // the last one advances it by the two steps.
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(a.g_done, 1u) == gridDim.x - 1) {
                *a.g_count = rec + 2;
                *a.g_done = 0;
            }
        }
    }
}

// The bookkeeping of two steps (linear_edge_kernel's, twice): boundary-flux
// sums of the interior lines from the pre-update momenta -- the input planes
// for the first step, the lines the pair kernel left for the second -- and
// domain%time (:117-205, :571).
template <typename R>
__global__ void __launch_bounds__(512) linear_pair_edge_kernel(const LinearPair<R> a, DevScalars *sc)
{
    const int nx = a.p.nx, ny = a.p.ny, n_ext = a.n_ext;
    const int64_t P = a.p.pitch;
    __shared__ double red[8][32];
    double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int i = n_ext + threadIdx.x; i <= nx - n_ext - 1; i += blockDim.x) {
        acc[0] += (double)a.p.vh[(int64_t)(ny - n_ext - 1) * P + i];
        acc[2] += (double)a.p.vh[(int64_t)(n_ext - 1) * P + i];
        acc[4] += (double)a.lines[i];
        acc[6] += (double)a.lines[nx + ny + i];
    }
    for (int r = n_ext + threadIdx.x; r <= ny - n_ext - 1; r += blockDim.x) {
        acc[1] += (double)a.p.uh[(int64_t)r * P + (nx - n_ext - 1)];
        acc[3] += (double)a.p.uh[(int64_t)r * P + (n_ext - 1)];
        acc[5] += (double)a.lines[nx + r];
        acc[7] += (double)a.lines[2 * nx + ny + r];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < 8; k++) {
        double v = acc[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL, v, o);
        if (lane == 0) red[k][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    const int nw = blockDim.x >> 5;
    for (int step = 0; step < 2; step++) {
        double s[4];
        for (int k = 0; k < 4; k++) {
            double v = 0.0;
            for (int w = 0; w < nw; w++) v += red[4 * step + k][w];
            s[k] = v;
        }
        const double time0 = sc->time;
        const double t_half = time0 + (double)(a.dt * K<R>::half());
        sc->boundary_flux_store[0] = s[0] * (double)a.m.dxb[ny - n_ext];
        sc->boundary_flux_store[1] = s[1] * (double)a.m.dyl[nx - n_ext];
        sc->boundary_flux_store[2] = -(s[2] * (double)a.m.dxb[n_ext]);
        sc->boundary_flux_store[3] = -(s[3] * (double)a.m.dyl[n_ext]);
        double tot = 0.0;
        for (int k = 0; k < 4; k++) tot += sc->boundary_flux_store[k];
        sc->boundary_flux_evolve_integral = tot * (double)a.dt;
        sc->boundary_flux_time_integral += sc->boundary_flux_evolve_integral;
        sc->time0 = time0;
        sc->time = t_half + (double)(K<R>::half() * a.dt);
        sc->dt = (double)a.dt;
        sc->dt_last_update = (double)a.dt;
        sc->evolve_step_dt = sc->time - time0;
        sc->nsteps_advanced += 1;
    }
}

template <typename R, bool COR, bool TL, bool NLF>
cudaError_t launch_pair(const LinearPair<R> &a, cudaStream_t s)
{
    constexpr int CPL = 16 / (int)sizeof(R);
    const int nstrips = (a.p.nx + 30 * CPL - 1) / (30 * CPL);
    const int sh = pair::rows((int64_t)nstrips * a.nbatch, a.p.ny, pair_warps(NLF, (int)sizeof(R)), NLF);
    const int64_t ctas = (int64_t)nstrips * ((a.p.ny + sh - 1) / sh) * a.nbatch;
    const size_t smem =
        16 * 32 * (NLF ? 7 : 5) * SLOTS + sizeof(RowConst<R>) * (sh + 4) + (a.g_n > 0 ? 4 * (sh + 5) : 0);
    auto go = [&](auto kernel) -> cudaError_t {
        return launch_behind(kernel, (unsigned)ctas, 32, smem, s, a, sh, nstrips);
    };
    if (a.g_n > 0) return go(linear_pair_kernel<R, COR, TL, NLF, true>);
    return go(linear_pair_kernel<R, COR, TL, NLF, false>);
}

}  // namespace

// Rows per segment (SWALS_PAIR_ROWS sets it): the count with the least
// estimate, over the rounds in which an SM takes its `resident` warps, of
//   (rows + 4) x sum of (A + warps of the round / 4),
// since a warp's row takes a time of its own (A) and its share of the
// scheduler's.  A is 3 for the first round and 1.5 for the next ones, whose
// warps start as others end; 2 for every round of the friction form.  Measured
// on the B200, us a step: 3600 x 2400 FP32 Coriolis 15 rows 37.4, 22 37.3, 33
// (1.2 rounds) 42.6, 41 (one round) 37.6, 48 39.6; 1200 x 800 FP64 Coriolis 8
// (1.1 rounds) 13.6, 10 10.9, 12 12.3, 16 11.9, 20 13.8; 400^2 FP64 2 5.5, 4
// 5.9, 6 7.0; friction 1501 x 1001 FP64 16 38.5, 20 (1.1 rounds) 42.3, 24 29.6,
// 32 34.4.  Beyond three rounds the HBM binds and 16 rows keep the rows that
// neighbours share in L2: 4096^2 FP32 14 59.7, 28 62.3, 64 70.1; FP64 16 112.1,
// 42 114.4, 85 120.0.
int pair::rows(int64_t strips, int ny, int resident, bool friction)
{
    const char *e = getenv("SWALS_PAIR_ROWS");
    if (e && atoi(e) > 0) return std::min(atoi(e), 256);
    static int sms = 0;
    if (sms == 0) {
        int dev = 0, n = 148;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms = n;
    }
    auto warps = [&](int sh) { return (double)strips * ((ny + sh - 1) / sh) / sms; };
    if (!friction && warps(16) > 3.0 * resident) return 16;
    int best = 0;
    double best_cost = 0.0;
    for (int sh = 2; sh <= 48; sh++) {
        double w = warps(sh), t = 0.0;
        for (double chain = friction ? 2.0 : 3.0; w > 0.0; w -= resident, chain = friction ? 2.0 : 1.5)
            t += chain + std::min(w, (double)resident) / 4.0;
        const double cost = (sh + 4.0) * t;
        if (best == 0 || cost < best_cost) {
            best = sh;
            best_cost = cost;
        }
    }
    return best;
}

template <typename R>
bool linear_pair_fits(const StepPlanes<R> &p, int64_t inst_stride, int64_t max_stride)
{
    const uintptr_t mis = (uintptr_t)p.stg | (uintptr_t)p.uh | (uintptr_t)p.vh | (uintptr_t)p.stg_o |
                          (uintptr_t)p.uh_o | (uintptr_t)p.vh_o | (uintptr_t)p.elv | (uintptr_t)p.max_stage |
                          (uintptr_t)(p.pitch * sizeof(R)) | (uintptr_t)(inst_stride * sizeof(R)) |
                          (uintptr_t)(max_stride * sizeof(R));
    return mis % 16 == 0 && p.nx >= 4 && p.ny >= 4;
}

template <typename R>
cudaError_t launch_linear_pair(LinearPair<R> a, const StepConfig &c, cudaStream_t s)
{
    a.xl = c.xl; a.xu = c.xu; a.yl = c.yl; a.yu = c.yu;
    a.msl = R(c.msl_linear);
    const R lfc = R(c.linear_friction_coeff);
    a.lin_fric = (lfc != R(0)) ? 1 : 0;
    a.lin_fric_mult = a.lin_fric ? (R(1) / (R(1) + a.dt * lfc)) : R(0);
    a.lin_fric_dt = a.dt * lfc;
    a.n_ext = c.exterior_cells_width;
    const bool cor = c.coriolis != 0;
    if (a.fw) {
        if (!c.truely_linear) return cudaErrorInvalidValue;   // the friction work changes every step
        return cor ? launch_pair<R, true, true, true>(a, s) : launch_pair<R, false, true, true>(a, s);
    }
    if (c.truely_linear) return cor ? launch_pair<R, true, true, false>(a, s) : launch_pair<R, false, true, false>(a, s);
    return cor ? launch_pair<R, true, false, false>(a, s) : launch_pair<R, false, false, false>(a, s);
}

template <typename R>
cudaError_t launch_linear_pair_edge(const LinearPair<R> &a0, const StepConfig &c, DevScalars *sc, cudaStream_t s)
{
    LinearPair<R> a = a0;
    a.n_ext = c.exterior_cells_width;
    linear_pair_edge_kernel<R><<<1, 512, 0, s>>>(a, sc);
    return cudaGetLastError();
}

#define SWALS_INST(R)                                                                             \
    template bool linear_pair_fits<R>(const StepPlanes<R> &, int64_t, int64_t);                   \
    template cudaError_t launch_linear_pair<R>(LinearPair<R>, const StepConfig &, cudaStream_t);  \
    template cudaError_t launch_linear_pair_edge<R>(const LinearPair<R> &, const StepConfig &, DevScalars *, cudaStream_t);
SWALS_INST(double)
SWALS_INST(float)

}  // namespace swals
