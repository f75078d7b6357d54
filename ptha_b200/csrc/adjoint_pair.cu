// adjoint_pair.cu -- two adjoint steps of the truly linear leapfrog in one
// pass over the grid: lambda <- M^T (C^T g' + M^T (C^T g + lambda)), with M^T as
// in adjoint.cu and C^T g the gauges' residuals added to lambda_STG.
//
// The transpose reaches one row and column either side like the step itself,
// so the pass is built like the forward pair (linear_pair.cu): a one-warp CTA
// owns 30 lanes x 16 bytes of columns plus a lane of halo either side and
// marches down a segment of rows plus two at each end, its rows arriving by
// 16-byte cp.async two rows ahead.  With row r of lambda and row r+1 of ELV:
//   face coefficients and total stage adjoint of row r, step 1's lambda_UH of
//   row r and lambda_VH of row r-1;
//   the same of step 2 one row above: lambda_STG and lambda_UH of row r-1 and
//   lambda_VH of row r-2 out.
// Each product that two cells or two rows share is formed once and comes by
// shuffle or in a register; the face coefficients serve both steps.  Products
// and sums keep the single step's operands and order: the same bits.
//
// A pass moves 56 B a cell (FP64) for two steps.  The single-step kernel is
// held by its 8-byte loads, shuffles and selects, not by memory.  Measured on
// the B200, us a step, that kernel / this one: 1200 x 800 FP64 Coriolis 22.8 /
// 10.1 (rows per segment one after another 6 12.8, 10 12.3, 16 13.8), 3600 x
// 2400 146 / 58 (4.2 TB/s), 1800 x 1200 FP32 32.8 / 12.9, 400^2 FP64 with 9
// gauges 12.3 / 4.0.
#include <type_traits>

#include "pair_common.cuh"

namespace swals {
namespace {

using pair::FULL;
using pair::cp16;

constexpr int SLOTS = 4;    // ring slots: row r, two in flight, and row r-1's ELV
constexpr int NP = 4;       // lambda_STG, lambda_UH, lambda_VH of row r, ELV of row r+1
constexpr int RESIDENT = 12;  // warps per SM (160 registers a thread)

template <typename R> __device__ __forceinline__ void cp_one(R *smem, const R *gmem, bool in)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(sa), "l"(gmem), "n"((int)sizeof(R)),
                 "r"(in ? (int)sizeof(R) : 0));
}

// Row constants: g dt/area, g dt/mean area, distance_bottom_edge(r + 1), the
// Coriolis factors of wet faces, dt/area, and dt/area x distance_bottom_edge
// of the row's south and north edge.
template <typename R> struct __align__(16) RowConst {
    R gu, gv, dxb1, cu, cv, cr, w0, w1;
};

template <typename R, bool COR>
__global__ void __launch_bounds__(32, RESIDENT) adjoint_pair_kernel(const AdjointPair<R> a, int SH, int nstrips)
{
    constexpr int CPL = 16 / (int)sizeof(R);
    constexpr int OUTC = 30 * CPL;
    typedef typename pair::Vec<R>::T V;
    extern __shared__ __align__(16) unsigned char pair_smem[];
    V *ring = reinterpret_cast<V *>(pair_smem);                               // [slot][plane][lane]
    R *beyond = reinterpret_cast<R *>(pair_smem + sizeof(V) * 32 * NP * SLOTS);   // [slot], 16 bytes each: ELV east of lane 31
    RowConst<R> *rc = reinterpret_cast<RowConst<R> *>(pair_smem + sizeof(V) * (32 * NP + 1) * SLOTS);
    const int lane = threadIdx.x;
    const int nx = a.nx, ny = a.ny;
    const int64_t P = a.P;
    const int strip = blockIdx.x % nstrips;
    const int ra = (blockIdx.x / nstrips) * SH, rb = min(ra + SH, ny);
    const R half = K<R>::half(), zero = K<R>::zero(), one = K<R>::one(), mad = K<R>::min_depth();
    const R dt = a.dt, msl = a.msl, mult = a.mult;

    for (int k = lane; k < rb - ra + 4; k += 32) {
        const int r = min(max(ra - 2 + k, 0), ny - 1);
        const R g = K<R>::gravity();
        RowConst<R> c;
        c.gu = g * dt / a.m.area[r];
        c.gv = g * dt / (half * (a.m.area[r] + a.m.area[min(r + 1, ny - 1)]));
        c.dxb1 = a.m.dxb[r + 1];
        c.cu = COR ? mult * (dt * a.m.cor[r] * half * one) * half : zero;
        c.cv = COR ? mult * (dt * a.m.cor_be[r + 1] * half * one) * half : zero;
        c.cr = dt / a.m.area[r];
        c.w0 = c.cr * a.m.dxb[r];
        c.w1 = c.cr * a.m.dxb[r + 1];
        rc[k] = c;
    }
    pair::GaugeRows gauges(reinterpret_cast<int *>(rc + (SH + 4)), a.sites, a.ng, ny, ra - 2, rb - ra + 4, lane);
    __syncwarp();
    gauges.ready(rb - ra + 4, lane);
    after_previous();   // (the metrics and gauge sites above are no kernel's output)
    let_next_start();

    const int c0 = strip * OUTC + (lane - 1) * CPL;          // this lane's first column
    const bool out = lane >= 1 && lane <= 30 && c0 < nx;
    const int src = c0 < 0 ? 0 : min(max(nx - c0, 0), CPL) * (int)sizeof(R);
    const int cl = src ? c0 : 0;                             // an address inside the row for zero-filled lanes
    const bool whole = c0 + CPL <= nx;
    const bool first = c0 == 0;
    const bool past = lane == 31 && c0 + CPL < nx;           // ELV of one more column
    R dyl[CPL + 1];
    unsigned im_m = 0u, is_m = 0u;                           // the columns in xL .. xU-1; in xL+1 .. xU-1 (one column more)
#pragma unroll
    for (int c = 0; c <= CPL; c++) {
        const int col = c0 + c;
        dyl[c] = a.m.dyl[min(max(col, 0), nx)];
        im_m |= (unsigned)(col >= a.xl && col <= a.xu - 1) << c;
        is_m |= (unsigned)(col >= a.xl + 1 && col <= a.xu - 1) << c;
    }
    // The gauges in the warp's columns, halo included; a cell may have several,
    // added in their order.
    auto inject = [&](int row, const double *resid, R(&s)[CPL]) {
        gauges.on_row(row - (ra - 2), strip * OUTC - CPL, strip * OUTC + OUTC + CPL - 1, lane,
                      [&](unsigned m, bool hit, int col, int q) {
            const R g = hit ? R(resid[q]) : zero;
            for (; m; m &= m - 1) {
                const int k = __ffs(m) - 1;
                const int at = __shfl_sync(FULL, col, k) - lane * CPL;
                const R gk = __shfl_sync(FULL, g, k);
#pragma unroll
                for (int c = 0; c < CPL; c++)
                    if (at == c) s[c] = s[c] + gk;
            }
        });
    };

    const int r0 = max(ra - 2, 0);
    auto issue = [&](int r, int slot) {
        if (r <= rb + 1) {
            V *s = ring + (size_t)slot * NP * 32 + lane;
            const int64_t o = (int64_t)min(r, ny - 1) * P + cl;
            const int n = r < ny ? src : 0;
            cp16(s, a.ls + o, n);
            cp16(s + 32, a.lu + o, n);
            cp16(s + 64, a.lv + o, n);
            const R *e = a.elv + (int64_t)min(r + 1, ny - 1) * P + cl;
            const int ne = r + 1 < ny ? src : 0;
            cp16(s + 96, e, ne);
            if (past) cp_one(beyond + slot * CPL, e + CPL, r + 1 < ny);
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
        o[0] = __shfl_up_sync(FULL, v[CPL - 1], 1);
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
    // march is in xL+1 .. xU-2, yL+1 .. yU-1, so nothing is selected.
    auto march = [&](auto inner) {
        constexpr bool INNER = decltype(inner)::value;
        struct Face { R aU[CPL], aV[CPL], cU[CPL], cV[CPL]; };
        // What a step leaves for the next row: total stage adjoint and
        // lambda_UH of the row, the part of its lambda_VH that the row itself
        // gives, and the products with the row's lambda_VH and stage adjoint.
        struct Row { R lst[CPL], lU[CPL], t[CPL], w[CPL], q[CPL], x[CPL]; };
        // One adjoint step at row r from its lambda (ls, lu, lv) and face
        // coefficients: row r's lst and lU, and lV of row r-1 into lv_s.  p: the
        // row before (after: this row).
        auto transpose = [&](int r, const RowConst<R> &k, const Face &f, const R(&ls)[CPL], const R(&lu)[CPL],
                             const R(&lv)[CPL], Row &p, R(&lv_s)[CPL]) {
            const bool im = r >= a.yl && r <= a.yu - 1;
            const bool is = r >= a.yl + 1 && r <= a.yu - 1;
            R pr[CPL], pw[CPL], x[CPL], xe[CPL], xse[CPL], y[CPL], yw[CPL], z[CPL], ze[CPL];
            Row n;
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                pr[c] = f.aU[c] * lu[c];
                n.q[c] = f.aV[c] * lv[c];
                n.x[c] = zero;
                if (COR) {
                    // V'(i, .) uses U(0, .) twice: 1/2 (U(0) + U(max(-1, 0)))
                    x[c] = (!INNER && c == 0 && first) ? f.cV[c] * R(2) * lv[c] : f.cV[c] * lv[c];
                    y[c] = f.cU[c] * lu[c];
                }
            }
            west(pr, pw);
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                n.lst[c] = ls[c] + pr[c] + n.q[c] - pw[c] - p.q[c];
                z[c] = k.cr * dyl[c] * n.lst[c];
            }
            east(z, ze);
            if (COR) {
                east(x, xe);
                east(p.x, xse);
                west(y, yw);
            }
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                const R idm = (INNER || (im && ((im_m >> c) & 1u))) ? mult : one;
                R lU = idm * lu[c], lV = idm * lv[c];
                R lS = p.t[c];                       // lV of the row before, so far
                if (COR) {
                    n.x[c] = x[c];
                    lU = lU - x[c];
                    lU = lU - xe[c];
                    lU = lU - p.x[c];
                    lU = lU - xse[c];
                    if (!INNER && r == 0) {
                        // U'(., 0) uses V(., 0) twice
                        lV = lV + R(2) * yw[c];
                        lV = lV + f.cU[c] * R(2) * lu[c];
                    } else {
                        lV = lV + yw[c];
                        lV = lV + y[c];
                    }
                    lS = lS + yw[c];
                    lS = lS + y[c];
                }
                if (INNER || (is && ((is_m >> c) & 1u))) lU = lU - z[c];
                if (INNER || (is && ((is_m >> (c + 1)) & 1u))) lU = lU + ze[c];
                if (INNER || (r - 1 >= a.yl + 1 && r - 1 <= a.yu - 1 && ((is_m >> c) & 1u))) lS = lS - p.w[c];
                if (INNER || (is && ((is_m >> c) & 1u))) lS = lS + k.w0 * n.lst[c];
                n.w[c] = k.w1 * n.lst[c];
                n.lU[c] = lU;
                n.t[c] = lV;
                lv_s[c] = lS;
            }
            p = n;
        };
        auto put = [&](R *plane, int row, const R(&x)[CPL]) {
            R *p = plane + (int64_t)row * P + c0;
            if (INNER || whole) {
                V v;
                R *vs = reinterpret_cast<R *>(&v);
#pragma unroll
                for (int c = 0; c < CPL; c++) vs[c] = x[c];
                *reinterpret_cast<V *>(p) = v;
            } else {
#pragma unroll
                for (int c = 0; c < CPL; c++)
                    if (c0 + c < nx) p[c] = x[c];
            }
        };

        Row A, B;          // of row r-1, step 1; of row r-2, step 2
        Face f1;           // of row r-1
        R e[CPL], e_last;  // ELV of row r
#pragma unroll
        for (int c = 0; c < CPL; c++) {
            A.lst[c] = A.lU[c] = A.t[c] = A.w[c] = A.q[c] = A.x[c] = zero;
            B.lst[c] = B.lU[c] = B.t[c] = B.w[c] = B.q[c] = B.x[c] = zero;
            f1.aU[c] = f1.aV[c] = f1.cU[c] = f1.cV[c] = zero;
            e[c] = (c0 + c >= 0 && c0 + c < nx) ? a.elv[(int64_t)r0 * P + c0 + c] : zero;
        }
        e_last = past ? a.elv[(int64_t)r0 * P + c0 + CPL] : zero;
        issue(r0, 0);
        issue(r0 + 1, 1);
#pragma unroll 1
        for (int r = r0, slot = 0; r <= rb + 1; r++, slot = (slot + 1) % SLOTS) {
            issue(r + 2, (slot + 2) % SLOTS);
            asm volatile("cp.async.wait_group 2;\n" ::);
            const V *s = ring + (size_t)slot * NP * 32 + lane;
            R ls[CPL], lu[CPL], lv[CPL], en[CPL], ee[CPL];
            get(s, 0, ls); get(s, 1, lu); get(s, 2, lv); get(s, 3, en);
            const RowConst<R> &k0 = rc[r - (ra - 2)];

            // Face coefficients of the momentum update (zero outside it).
            Face f;
            east(e, ee);
            if (lane == 31) ee[CPL - 1] = e_last;
            {
                const R lim = -mad + msl;
                const bool im = r >= a.yl && r <= a.yu - 1;
                const R cu0 = k0.cu * zero, cv0 = k0.cv * zero;
#pragma unroll
                for (int c = 0; c < CPL; c++) {
                    const bool in = INNER || (im && ((im_m >> c) & 1u));
                    const bool w0 = e[c] < lim;
                    const R hU = (w0 && ee[c] < lim) ? fma(-half, ee[c] + e[c], msl) : zero;
                    const R hV = (en[c] < lim && w0) ? fma(-half, en[c] + e[c], msl) : zero;
                    const R aU = mult * (k0.gu * hU * dyl[c + 1]);
                    const R aV = mult * (k0.gv * hV * k0.dxb1);
                    f.aU[c] = in ? aU : zero;
                    f.aV[c] = in ? aV : zero;
                    f.cU[c] = in ? ((hU > zero) ? k0.cu : cu0) : zero;
                    f.cV[c] = in ? ((hV > zero) ? k0.cv : cv0) : zero;
                }
            }
            // step 1 at row r, step 2 at row r-1
            R lsB[CPL], luB[CPL], lvB[CPL], lvo[CPL];
#pragma unroll
            for (int c = 0; c < CPL; c++) { lsB[c] = A.lst[c]; luB[c] = A.lU[c]; }
            // (one rare branch for both steps: with one before each, 3600 x 2400
            // takes 61.8 us a step, 2400 x 1600 30.2, with this 60.3 and 27.0)
            if (gauges.on(r - (ra - 2)) || gauges.on(r - (ra - 1))) {
                inject(r, a.resid, ls);
                if (r > r0) inject(r - 1, a.resid2, lsB);
            }
            transpose(r, k0, f, ls, lu, lv, A, lvB);
            if (r > r0) {
                transpose(r - 1, rc[r - 1 - (ra - 2)], f1, lsB, luB, lvB, B, lvo);
                if (out) {
                    if (r - 1 >= ra && r - 1 < rb) { put(a.ls_o, r - 1, B.lst); put(a.lu_o, r - 1, B.lU); }
                    if (r - 2 >= ra) put(a.lv_o, r - 2, lvo);
                }
            }
            f1 = f;
#pragma unroll
            for (int c = 0; c < CPL; c++) e[c] = en[c];
            e_last = beyond[slot * CPL];
        }
        asm volatile("cp.async.wait_group 0;\n" ::);
    };
    // Columns strip * OUTC - CPL .. (strip + 1) * OUTC + CPL and rows ra - 2 .. rb + 1.
    if (strip * OUTC - CPL >= a.xl + 1 && (strip + 1) * OUTC + CPL <= a.xu - 1 && ra - 2 >= a.yl + 1 && rb + 1 <= a.yu - 1)
        march(std::true_type());
    else
        march(std::false_type());
}

}  // namespace

template <typename R>
cudaError_t launch_adjoint_pair(const AdjointPair<R> &a, bool coriolis, cudaStream_t s)
{
    constexpr int CPL = 16 / (int)sizeof(R);
    const int nstrips = (a.nx + 30 * CPL - 1) / (30 * CPL);
    const int sh = pair::rows(nstrips, a.ny, RESIDENT, false);
    const unsigned ctas = (unsigned)(nstrips * ((a.ny + sh - 1) / sh));
    const size_t smem = 16 * (32 * NP + 1) * SLOTS + sizeof(RowConst<R>) * (sh + 4) + (a.ng > 0 ? 4 * (sh + 5) : 0);
    if (coriolis) return launch_behind(adjoint_pair_kernel<R, true>, ctas, 32, smem, s, a, sh, nstrips);
    return launch_behind(adjoint_pair_kernel<R, false>, ctas, 32, smem, s, a, sh, nstrips);
}
template cudaError_t launch_adjoint_pair<double>(const AdjointPair<double> &, bool, cudaStream_t);
template cudaError_t launch_adjoint_pair<float>(const AdjointPair<float> &, bool, cudaStream_t);

}  // namespace swals
