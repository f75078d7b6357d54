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
// A warp owns a strip of 30 lanes x 16 bytes (60 FP64 or 120 FP32 columns)
// plus one lane of halo either side -- two steps reach two columns, and a lane
// holds at least two -- and marches down a segment of rows plus two at each
// end.  When row r arrives (by 16-byte cp.async, two rows ahead):
//   stage of step 1 in row r, momenta of step 1 in row r-1,
//   stage of step 2 in row r-1, momenta of step 2 in row r-2, row r-2 out.
// What a row still needs of the rows before stays in registers, neighbouring
// columns come by shuffle, and there is no barrier in the march.  Both steps
// are written with the expressions of the single step, in their order, so the
// results are the same bits.  The row constants (dt / area and so on) are
// formed once per segment row in shared memory, the face depths of the truly
// linear solver once for both steps.
//
// 16-byte lanes start on 16-byte boundaries (strips every 480 bytes, 15 whole
// sectors); planes that linear_pair_fits refuses step one at a time.
//
// Measured on the B200, us a step, one step at a time / in pairs: 4096^2 FP64
// 212 / 118, 8192^2 791 / 421 (a pair moves 72 B a cell: 5.1 and 5.7
// TB/s, 0.79 and 0.89 of the copy bandwidth), 3600 x 2400 FP32 Coriolis 71.8 /
// 43.6, 1200 x 800 Coriolis 20.5 / 12.2, 400^2 with 9 gauges 9.2 / 6.4, 200 x
// 150 9.3 / 4.9; with Manning friction 1501 x 1001 Coriolis 58.1 / 29.3.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "swals_kernels.h"

namespace swals {
namespace {

constexpr int WPC = 4;      // warps (strips) per CTA
constexpr int SLOTS = 3;    // ring slots per warp (two rows in flight)
constexpr unsigned FULL = 0xffffffffu;

template <typename R> struct Vec;
template <> struct Vec<double> { typedef double2 T; };
template <> struct Vec<float> { typedef float4 T; };

__device__ __forceinline__ void cp16(void *smem, const void *gmem, int src_bytes)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(src_bytes));
}

// CTAs per SM the register cap is sized for.  With the friction work the two
// steps' square roots and quotients bind, not the memory, and spills cost more
// than warps: 1501 x 1001 FP64 Coriolis 52.3 us a step at 4 (spilling), 29.5
// at 3, 29.3 at 2 (188 registers); FP32 3000 x 2000 95 / 77 / 77.
constexpr int pair_ctas(bool nlf, int real_bytes) { return !nlf ? 4 : real_bytes == 8 ? 2 : 3; }

// Row constants of a segment, rows ra - 2 .. (clamped to the grid).
template <typename R> struct RowConst {
    R cs, cu, cv, dxb, dxb1, dtc, dtj;   // dt/area, g dt/area, g dt/mean area, distance_bottom_edge(r), (r+1), dt cor/2 ...
};

template <typename R, bool COR, bool TL, bool NLF, bool GAUGES>
__global__ void __launch_bounds__(32 * WPC, pair_ctas(NLF, (int)sizeof(R))) linear_pair_kernel(const LinearPair<R> a, int SH, int nstrips)
{
    constexpr int CPL = 16 / (int)sizeof(R);
    constexpr int OUTC = 30 * CPL;
    constexpr int NP = NLF ? 7 : 5;      // UH, VH, STG, ELV, max_stage (of row r-2), friction work at UH, VH
    constexpr bool AVG = COR || NLF;     // the two-point averages of the other momentum
    typedef typename Vec<R>::T V;
    extern __shared__ __align__(16) unsigned char pair_smem[];
    RowConst<R> *rc = reinterpret_cast<RowConst<R> *>(pair_smem + sizeof(V) * 32 * NP * SLOTS * WPC);
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    V *ring = reinterpret_cast<V *>(pair_smem) + (size_t)wib * SLOTS * NP * 32;   // [slot][plane][lane]

    const int nx = a.p.nx, ny = a.p.ny;
    const int64_t P = a.p.pitch;
    const int b = blockIdx.x % a.nbatch;               // instance: neighbouring CTAs share ELV rows in L2
    const int tile = blockIdx.x / a.nbatch;
    const int groups = (nstrips + WPC - 1) / WPC;
    const int strip = (tile % groups) * WPC + wib;
    const int ra = (tile / groups) * SH;
    const int rb = min(ra + SH, ny);
    const R half = K<R>::half(), zero = K<R>::zero(), one = K<R>::one(), mad = K<R>::min_depth();
    const R dt = a.dt, msl = a.msl;

    for (int k = threadIdx.x; k < rb - ra + 4; k += 32 * WPC) {
        const int r = min(max(ra - 2 + k, 0), ny - 1);
        const R g = K<R>::gravity();
        RowConst<R> c;
        c.cs = dt / a.m.area[r];
        c.cu = g * dt / a.m.area[r];
        c.cv = g * dt / (half * (a.m.area[r] + a.m.area[min(r + 1, ny - 1)]));
        c.dxb = a.m.dxb[r];
        c.dxb1 = a.m.dxb[r + 1];
        c.dtc = COR ? dt * a.m.cor[r] * half : zero;
        c.dtj = COR ? dt * a.m.cor_be[r + 1] * half : zero;
        rc[k] = c;
    }
    __syncthreads();
    const int rec = GAUGES ? (a.g_count ? *a.g_count : 0) : 0;

    if (strip < nstrips) {
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
        // gauges in this lane's own columns (up to 64 sites; more are looked up cell by cell)
        unsigned long long gm = 0ull;
        if (GAUGES && out)
            for (int q = 0; q < min(a.g_n, 64); q++)
                if (a.g_sites[2 * q] >= c0 && a.g_sites[2 * q] < c0 + CPL && a.g_sites[2 * q + 1] >= ra &&
                    a.g_sites[2 * q + 1] < rb)
                    gm |= 1ull << q;
        auto record = [&](int step, int row, const R(&s)[CPL], const R(&u)[CPL], const R(&v)[CPL]) {
            if (rec + step >= a.g_capacity) return;
            auto put = [&](int q) {
#pragma unroll
                for (int c = 0; c < CPL; c++)
                    if (a.g_sites[2 * q] == c0 + c && a.g_sites[2 * q + 1] == row) {
                        double *d = a.g_rec + (((int64_t)(rec + step) * a.nbatch + b) * a.g_n + q) * a.g_vals;
                        d[0] = (double)s[c];
                        if (a.g_vals == 3) { d[1] = (double)u[c]; d[2] = (double)v[c]; }
                    }
            };
            if (a.g_n > 64) {
                if (out)
                    for (int q = 0; q < a.g_n; q++)
                        if (a.g_sites[2 * q + 1] == row) put(q);
            } else {
                for (unsigned long long m = gm; m; m &= m - 1) put(__ffsll((long long)m) - 1);
            }
        };
        // the lane's component on the west and east boundary-flux lines, or -1
        const int ln_e = (a.lines && out) ? nx - a.n_ext - 1 - c0 : -1, ln_w = (a.lines && out) ? a.n_ext - 1 - c0 : -1;

        const int r0 = max(ra - 2, 0);
        auto issue = [&](int r) {
            if (r <= rb + 1) {
                V *s = ring + (size_t)((r - r0) % SLOTS) * NP * 32 + lane;
                const int rr = min(r, ny - 1);
                const int64_t o = (int64_t)rr * P + cl;
                const int n = r < ny ? src : 0;
#pragma unroll
                for (int k = 0; k < 4; k++) cp16(s + k * 32, pl[k] + o, n);
                const bool mx = max_stage && r - 2 >= ra && out;
                cp16(s + 4 * 32, mx ? max_stage + (int64_t)(r - 2) * P + cl : pl[2] + o, mx ? src : 0);
                if (NLF) {
                    cp16(s + 5 * 32, a.fw + o, n);
                    cp16(s + 6 * 32, a.fw + a.fw_plane + o, n);
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
        // New stage of row r (:92-115).
        auto stage = [&](int r, const RowConst<R> &k, const R(&s)[CPL], const R(&u)[CPL], const R(&uw)[CPL],
                         const R(&v)[CPL], const R(&vs)[CPL], R(&o)[CPL]) {
            const bool row = r >= a.yl + 1 && r <= a.yu - 1;
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                const R t1 = (u[c] - uw[c]) * dyl[c];
                const R t2 = v[c] * k.dxb1 - vs[c] * k.dxb;
                const R n = s[c] - k.cs * (t1 + t2);
                o[c] = (row && ((st_m >> c) & 1u)) ? n : s[c];
            }
        };
        // Face depths (:353-370); not truly linear: of the new stage.
        auto depths = [&](const R(&e)[CPL], const R(&ee)[CPL], const R(&en)[CPL], const R(&s)[CPL], const R(&se)[CPL],
                          const R(&sn)[CPL], R(&hi)[CPL], R(&hj)[CPL]) {
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                if (TL) {
                    const R lim = -mad + msl;
                    const bool w0 = e[c] < lim;
                    hi[c] = (w0 && ee[c] < lim) ? (msl - half * (ee[c] + e[c])) : zero;
                    hj[c] = (en[c] < lim && w0) ? (msl - half * (en[c] + e[c])) : zero;
                } else {
                    const bool w0 = s[c] - e[c] > mad;
                    hi[c] = (w0 && se[c] - ee[c] > mad) ? (half * ((se[c] + s[c]) - (ee[c] + e[c]))) : zero;
                    hj[c] = (sn[c] - en[c] > mad && w0) ? (half * ((sn[c] + s[c]) - (en[c] + e[c]))) : zero;
                }
            }
        };
        // Momenta of row j (:225-567) from the old momenta u, v (rows j; vs:
        // VH of row j-1, un / uwn: UH of row j+1 and its west neighbour) and
        // the new stage s, se, sn.
        auto momenta = [&](int j, const RowConst<R> &k, const R(&u)[CPL], const R(&v)[CPL], const R(&s)[CPL],
                           const R(&se)[CPL], const R(&sn)[CPL], const R(&hi)[CPL], const R(&hj)[CPL],
                           const R(&vs)[CPL], const R(&uw)[CPL], const R(&un)[CPL], const R(&uwn)[CPL],
                           const R(&fu)[CPL], const R(&fv)[CPL], R(&ou)[CPL], R(&ov)[CPL]) {
            const bool row = j >= a.yl && j <= a.yu - 1;
            R ve[CPL], vse[CPL], vsc[CPL];
            if (AVG) {
#pragma unroll
                for (int c = 0; c < CPL; c++) vsc[c] = (j == 0) ? v[c] : vs[c];
                east(v, ve);
                east(vsc, vse);
            }
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                R uu = u[c], vv = v[c];
                if (!TL) {   // wet factors
                    uu = uu * ((hi[c] > zero) ? one : zero);
                    vv = vv * ((hj[c] > zero) ? one : zero);
                }
                uu = uu - k.cu * hi[c] * (se[c] - s[c]) * dyl[c + 1];
                vv = vv - k.cv * hj[c] * (sn[c] - s[c]) * k.dxb1;
                if (AVG) {
                    const R vh_iph_jmh = half * (vsc[c] + vse[c]);
                    const R vh_iph_jph = half * (v[c] + ve[c]);
                    const R uh_i_j = half * (u[c] + uw[c]);
                    const R uh_i_jp1 = half * (un[c] + uwn[c]);
                    if (COR) {
                        uu = uu + k.dtc * ((hi[c] > zero) ? one : zero) * (vh_iph_jmh + vh_iph_jph);
                        vv = vv - k.dtj * ((hj[c] > zero) ? one : zero) * (uh_i_j + uh_i_jp1);
                    }
                    if (NLF) {
                        const R tv = half * (vh_iph_jmh + vh_iph_jph);
                        const R tu = half * (uh_i_j + uh_i_jp1);
                        uu = friction_multiplier(one + a.lin_fric_dt, dt, fu[c], u[c], tv) * uu;
                        vv = friction_multiplier(one + a.lin_fric_dt, dt, fv[c], v[c], tu) * vv;
                    }
                }
                if (!NLF && a.lin_fric) {
                    uu = a.lin_fric_mult * uu;
                    vv = a.lin_fric_mult * vv;
                }
                const bool ok = row && ((mo_m >> c) & 1u);
                ou[c] = ok ? uu : u[c];
                ov[c] = ok ? vv : v[c];
            }
        };

        // Of row r-1: ELV, old UH (and its west neighbour), old VH, stage of
        // step 1; of row r-2: VH; stage of step 1, momenta of step 1, stage of
        // step 2, face depths; of row r-3: VH of step 1.
        R e1[CPL], u1[CPL], v1[CPL], a1[CPL], uw1[CPL], v2[CPL], f1[CPL], g1[CPL];
        R a2[CPL], uA2[CPL], vA2[CPL], b2[CPL], hi2[CPL], hj2[CPL], vA3[CPL], uAw2[CPL], f2[CPL], g2[CPL], e2[CPL];
#pragma unroll
        for (int c = 0; c < CPL; c++) {
            e1[c] = u1[c] = v1[c] = a1[c] = uw1[c] = v2[c] = f1[c] = g1[c] = zero;
            a2[c] = uA2[c] = vA2[c] = b2[c] = hi2[c] = hj2[c] = vA3[c] = uAw2[c] = f2[c] = g2[c] = e2[c] = zero;
        }
        for (int r = r0; r < r0 + SLOTS - 1; r++) issue(r);
        for (int r = r0; r <= rb + 1; r++) {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(SLOTS - 2));
            const V *s = ring + (size_t)((r - r0) % SLOTS) * NP * 32 + lane;
            R u[CPL], v[CPL], st[CPL], e[CPL], mx[CPL], f[CPL], g[CPL];
            get(s, 0, u); get(s, 1, v); get(s, 2, st); get(s, 3, e); get(s, 4, mx);
#pragma unroll
            for (int c = 0; c < CPL; c++) f[c] = g[c] = zero;
            if (NLF) { get(s, 5, f); get(s, 6, g); }
            issue(r + SLOTS - 1);   // (into the slot read in the iteration before)
            const RowConst<R> &k0 = rc[r - (ra - 2)];
            const RowConst<R> &k1 = rc[max(r - 1 - (ra - 2), 0)];
            const RowConst<R> &k2 = rc[max(r - 2 - (ra - 2), 0)];

            // step 1: stage of row r, momenta of row r-1
            R uw[CPL], sA[CPL], ae[CPL], ee[CPL], hi[CPL], hj[CPL], uA[CPL], vA[CPL];
            west(u, uw);
            stage(r, k0, st, u, uw, v, v1, sA);
            east(a1, ae);
            east(e1, ee);
            depths(e1, ee, e, a1, ae, sA, hi, hj);
            momenta(r - 1, k1, u1, v1, a1, ae, sA, hi, hj, v2, uw1, u, uw, f1, g1, uA, vA);
            if (GAUGES && r - 1 >= ra && r - 1 < rb) record(0, r - 1, a1, uA, vA);
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
            R uAw[CPL], sB[CPL], be[CPL], uB[CPL], vB[CPL];
            west(uA, uAw);
            stage(r - 1, k1, a1, uA, uAw, vA, vA2, sB);
            east(b2, be);
            if (!TL) {
                R e2e[CPL];
                east(e2, e2e);
                depths(e2, e2e, e1, b2, be, sB, hi2, hj2);
            }
            momenta(r - 2, k2, uA2, vA2, b2, be, sB, hi2, hj2, vA3, uAw2, uA, uAw, f2, g2, uB, vB);

            const int q = r - 2;
            if (q >= ra && out) {   // (r <= rb + 1)
                const int64_t o = (int64_t)q * P + c0;
                const bool my = max_stage && q >= a.yl && q <= a.yu;
                R m[CPL];
#pragma unroll
                for (int c = 0; c < CPL; c++) {
                    const R t = (a2[c] > mx[c]) ? a2[c] : mx[c];
                    m[c] = (my && ((ms_m >> c) & 1u)) ? ((b2[c] > t) ? b2[c] : t) : mx[c];
                }
                if (whole) {
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
                if (GAUGES) record(1, q, b2, uB, vB);
            }
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                e2[c] = e1[c]; e1[c] = e[c];
                v2[c] = v1[c]; u1[c] = u[c]; v1[c] = v[c]; uw1[c] = uw[c];
                a2[c] = a1[c]; a1[c] = sA[c];
                vA3[c] = vA2[c]; uA2[c] = uA[c]; vA2[c] = vA[c]; uAw2[c] = uAw[c];
                b2[c] = sB[c]; hi2[c] = hi[c]; hj2[c] = hj[c];
                f2[c] = f1[c]; g2[c] = g1[c]; f1[c] = f[c]; g1[c] = g[c];
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::);
    }

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

// Rows per segment (SWALS_PAIR_ROWS sets it): the candidate with the least
// estimate of
//   (rows + 3) x CTA-rows that an SM works through per row of a segment,
// as for the finite-volume strips (fv_rows): up to five CTAs of an SM side by
// side, fewer than two and a half taking the time of two and a half (a row of
// one CTA is a chain of 1.2 us for the two steps at 400 x 400, against 0.45 us
// a CTA-row on full SMs).  Measured on the B200, us a step, the estimate's
// rows (best of 4 .. 64): 200 x 150 FP64 4: 4.9; 400^2 4: 6.4; 1200 x 800
// Coriolis 8: 12.2 (16: 11.8); 4096^2 64: 118.1 (24: 112.7); 8192^2 48:
// 420.7; 3600 x 2400 FP32 Coriolis 48: 43.6.
// The friction form runs two (FP32 three) CTAs an SM in equal rounds: 24 rows
// at 1501 x 1001, the best there.
int pair_rows(int64_t groups, int ny, int nbatch, int rounds_of)
{
    const char *e = getenv("SWALS_PAIR_ROWS");
    if (e && atoi(e) > 0) return std::min(atoi(e), 256);
    static int sms = 0;
    if (sms == 0) {
        int dev = 0, n = 148;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms = n;
    }
    constexpr double resident = 5.0, chain = 2.5;
    int best = 0;
    double best_cost = 0.0;
    for (int sh : {4, 6, 8, 12, 16, 24, 32, 48, 64}) {
        const double ctas = (double)groups * nbatch * ((ny + sh - 1) / sh) / sms;
        double w;
        if (rounds_of) {
            w = rounds_of * std::ceil(ctas / rounds_of);
        } else if (ctas <= resident) {
            w = std::max(chain, std::ceil(ctas));
        } else {
            const double rest = std::fmod(ctas, resident);
            w = ctas + (rest > 0.0 ? std::max(chain - rest, 0.0) : 0.0);
        }
        const double cost = (sh + 3.0) * w;
        if (best == 0 || cost < best_cost) {
            best = sh;
            best_cost = cost;
        }
    }
    return best;
}

template <typename R, bool COR, bool TL, bool NLF>
cudaError_t launch_pair(const LinearPair<R> &a, cudaStream_t s)
{
    constexpr int CPL = 16 / (int)sizeof(R);
    const int nstrips = (a.p.nx + 30 * CPL - 1) / (30 * CPL);
    const int64_t groups = (nstrips + WPC - 1) / WPC;
    const int sh = pair_rows(groups, a.p.ny, a.nbatch, NLF ? pair_ctas(NLF, (int)sizeof(R)) : 0);
    const int64_t ctas = groups * ((a.p.ny + sh - 1) / sh) * a.nbatch;
    const size_t smem = 16 * 32 * (NLF ? 7 : 5) * SLOTS * WPC + sizeof(RowConst<R>) * (sh + 4);
    auto go = [&](auto kernel) -> cudaError_t {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
        if (e != cudaSuccess) return e;
        kernel<<<(unsigned)ctas, 32 * WPC, smem, s>>>(a, sh, nstrips);
        return cudaGetLastError();
    };
    if (a.g_n > 0) return go(linear_pair_kernel<R, COR, TL, NLF, true>);
    return go(linear_pair_kernel<R, COR, TL, NLF, false>);
}

}  // namespace

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
