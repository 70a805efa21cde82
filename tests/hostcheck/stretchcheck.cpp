// Test-only host build: element matrices in the FS_FP64 fixed point
// (csrc/fs_elem_fixed.cuh) and in double (csrc/fs_elem_math.cuh), less the same in
// long double (wide_elem_math.h, the latter header with every double widened).
// Not part of the product.
#include <stdint.h>
#include <string.h>

#include <algorithm>

#include "fs_host_prep.h"
#include "fs_elem_fixed.cuh"
#include "wide_elem_math.h"

using namespace fs;

template <class E, int NN = 3> static E element(const double *X, const double *nrm, double t)
{
    E in;
    memset(&in, 0, sizeof in);
    for (int a = 0; a < NN; a++) {
        for (int c = 0; c < 3; c++) {
            in.X[a][c] = X[3 * a + c];
            in.nrm[a][c] = nrm[3 * a + c];
        }
        in.valid[a] = true;
    }
    in.t = t;
    return in;
}

// node blocks from expanded rows
template <int NP, int NN, int MS, int BS, int BSS, int DR>
static void blocks(FxSlots rows, int step, const FxExp &ex, double *K)
{
    for (int p = 0; p < NN; p++)
        for (int q = 0; q < NN; q++) {
            double o[3][6], b[3][6];
            if (p == q) {
                fx_block_top<NP, MS, BS, BSS, true>(rows, step, p, q, ex, o);
                fx_block_bottom<NP, BS, BSS, true>(rows, step, p, q, rows + (DR + 3 * p), ex, b);
                for (int i = 0; i < 3; i++)
                    for (int j = 0; j < 3; j++) b[i][j] = o[j][3 + i];
            } else {
                fx_block_top<NP, MS, BS, BSS, false>(rows, step, p, q, ex, o);
                fx_block_bottom<NP, BS, BSS, false>(rows, step, p, q, rows, ex, b);
            }
            for (int i = 0; i < 3; i++)
                for (int j = 0; j < 6; j++) {
                    K[(6 * p + i) * 6 * NN + 6 * q + j] = o[i][j];
                    K[(6 * p + 3 + i) * 6 * NN + 6 * q + j] = b[i][j];
                }
        }
}

// the outputs of one element: the long double matrix (rounded) and the differences
// of the fixed point's, F, and of the double rows' from it
static void compare(int nd, int nrows, const double *F, const double *rows, const long double *wide, double *K,
                    double *dfixed, double *ddouble)
{
    for (int i = 0; i < nd; i++)
        for (int j = 0; j < nd; j++) {
            double d = 0;
            long double s = 0;
            for (int r = 0; r < nrows; r++) {
                d = fma(rows[nd * r + i], rows[nd * r + j], d);
                s += wide[nd * r + i] * wide[nd * r + j];
            }
            K[nd * i + j] = (double)s;
            dfixed[nd * i + j] = (double)(F[nd * i + j] - s);
            ddouble[nd * i + j] = (double)(d - s);
        }
}

static int constants(const fs_shell_params &p, MatConst &mc, fsl::MatConst &ml)
{
    if (prepare_matconst(p, mc)) return 1;
    memset(&ml, 0, sizeof ml);
    for (int i = 0; i < 6; i++) ml.Lps[i] = mc.Lps[i];
    for (int i = 0; i < 3; i++) ml.Lt[i] = mc.Lt[i];
    ml.stab_c = mc.stab_c;
    ml.drill_scale = mc.drill_scale;
    return 0;
}

extern "C" {

// n triangles: X, nrm (3 x 3 each), t; of each, 18 x 18: the long double matrix
// (rounded), the fixed point's and the double's difference from it; whether it is
// left to the double kernel
int stretched_triangles(int64_t n, const double *X, const double *nrm, const double *t, const fs_shell_params *p,
                        double *K, double *dfixed, double *ddouble, uint8_t *elongated)
{
    MatConst mc;
    fsl::MatConst ml;
    if (constants(*p, mc, ml)) return 1;
    typedef CompactRows<3, 2> L;
    static FxSlot mem[(L::SIZE + 1) * FX_GROUP];
    const FxSlots slot{mem};
    for (int64_t e = 0; e < n; e++) {
        const ElemIn<3> in = element<ElemIn<3>>(X + 9 * e, nrm + 9 * e, t[e]);
        const fsl::ElemIn<3> il = element<fsl::ElemIn<3>>(X + 9 * e, nrm + 9 * e, t[e]);
        double rows[11 * 18], F[324];
        long double wide[11 * 18];
        t3_rows<double, false, false>(in, mc, nullptr, rows, 18);
        fsl::t3_rows<long double, false, false>(il, ml, nullptr, wide, 18);
        FxGeom<3> geo;
        FxMax mx;
        elongated[e] = t3_coefs(in, mc, slot, geo, mx);
        if (!mx.usable()) return 2;
        const FxExp ex = fx_exponents(mx, 0);
        t3_expand(slot, geo, in.valid, ex);
        blocks<1, 3, L::MS, L::BS, L::BSS, L::DR>(slot, 0, ex, F);
        compare(18, 11, F, rows, wide, K + 324 * e, dfixed + 324 * e, ddouble + 324 * e);
    }
    return 0;
}

// the same of n quadrilaterals (4 x 3 each, 24 x 24)
int stretched_quads(int64_t n, const double *X, const double *nrm, const double *t, const fs_shell_params *p, double *K,
                    double *dfixed, double *ddouble)
{
    MatConst mc;
    fsl::MatConst ml;
    if (constants(*p, mc, ml)) return 1;
    typedef Q4Compact L;
    static FxSlot mem[(L::SIZE + 1) * FX_GROUP];
    const FxSlots slot{mem};
    for (int64_t e = 0; e < n; e++) {
        const ElemIn<4> in = element<ElemIn<4>, 4>(X + 12 * e, nrm + 12 * e, t[e]);
        const fsl::ElemIn<4> il = element<fsl::ElemIn<4>, 4>(X + 12 * e, nrm + 12 * e, t[e]);
        Q4Elem qe;
        fsl::Q4Elem ql;
        q4_prepare(in, in.t, mc.stab_c, qe);
        fsl::q4_prepare(il, il.t, ml.stab_c, ql);
        double rows[36 * 24], F[576], td[4] = {0, 0, 0, 0}, tp[4], tr[4] = {0, 0, 0, 0}, rn[4], sum = 0;
        long double wide[36 * 24], tl[4] = {0, 0, 0, 0}, tq[4];
        FxGeom<4> geo[4];
        FxMax mx;
        for (int k = 0; k < 4; k++) rn[k] = 1.0 / sqrt(dot3(in.nrm[k], in.nrm[k]));
        for (int j = 0; j < 4; j++) {
            if (q4_coefs(qe.Xr, in.nrm, in.valid, rn, in.t, sqrt(qe.stab), j, mc, slot + j * L::GP, geo[j], mx, tp)) return 2;
            for (int k = 0; k < 4; k++) tr[k] += tp[k];
            q4_point_rows<double, false>(in, qe, j, mc, nullptr, rows + j * 8 * 24, 24, tp);
            for (int k = 0; k < 4; k++) td[k] += tp[k];
            fsl::q4_point_rows<long double, false>(il, ql, j, ml, nullptr, wide + j * 8 * 24, 24, tq);
            for (int k = 0; k < 4; k++) tl[k] += tq[k];
        }
        q4_drill_rows<double>(in, td, mc.drill_scale, rows + 32 * 24, 24);
        fsl::q4_drill_rows<long double>(il, tl, ml.drill_scale, wide + 32 * 24, 24);
        for (int k = 0; k < 4; k++) sum += tr[k] > 0.0 ? tr[k] / 2 : 0.0;
        const double sk = sqrt(sum / 4 * mc.drill_scale);
        for (int k = 0; k < 12; k++) fx_max(mx.r, sk * in.nrm[k / 3][k % 3]);
        if (!mx.usable()) return 3;
        const FxExp ex = fx_exponents(mx, 1);
        for (int j = 0; j < 4; j++) {
            fx ax[4][3][3];
            expand_slots<4, L::MS, L::BS, L::BSS>(slot + j * L::GP, geo[j], ex, ax);
        }
        for (int k = 0; k < 12; k++) slot[L::DR + k].x = fx_make(sk * in.nrm[k / 3][k % 3], ex.r);
        blocks<4, 4, L::MS, L::BS, L::BSS, L::DR>(slot, L::GP, ex, F);
        compare(24, 36, F, rows, wide, K + 576 * e, dfixed + 576 * e, ddouble + 576 * e);
    }
    return 0;
}

}  // extern "C"

// a layered element's rows (NR dense ones, then the drilling rows' rotations) to
// fixed point and multiplied, as the kernels do
template <int NN, int NR> static bool layered_blocks(double *rows, int spare, double *K)
{
    typedef LayeredRows<NN, NR> L;
    DofMax<NN> mx;
    mx.zero();
    for (int k = 0; k < NR; k++) mx.row(rows + k * L::RS);
    for (int k = 0; k < 3 * NN; k++) fx_max(mx.m[k / 3][3 + k % 3], rows[L::DR + k]);
    if (!mx.usable()) return false;
    DofExp E[NN];
    for (int a = 0; a < NN; a++) {
        E[a] = mx.exponents(a, spare);
        for (int k = 0; k < NR; k++)
            for (int q = 0; q < 6; q++) to_fixed(rows + L::RS * k + 6 * a + q, dof_exp(E[a], q));
        for (int q = 0; q < 3; q++) to_fixed(rows + L::DR + 3 * a + q, dof_exp(E[a], 3 + q));
    }
    for (int a = 0; a < NN; a++)
        for (int b = 0; b < NN; b++) {
            double t[3][6], u[3][6];
            if (a == b) {
                fixed_rows<NR, L::RS, true, 0>(rows, rows + L::DR + 3 * a, a, a, E[a], E[a], t);
                fixed_rows<NR, L::RS, true, 3>(rows, rows + L::DR + 3 * a, a, a, E[a], E[a], u);
                for (int i = 0; i < 3; i++)
                    for (int j = 0; j < 3; j++) {
                        if (j < i) t[i][j] = t[j][i];
                        u[i][j] = t[j][3 + i];
                        if (j < i) u[i][3 + j] = u[j][3 + i];
                    }
            } else {
                fixed_rows<NR, L::RS, false, 0>(rows, rows, a, b, E[a], E[b], t, 0);
                fixed_rows<NR, L::RS, false, 0>(rows, rows, a, b, E[a], E[b], u, 3);
            }
            for (int i = 0; i < 3; i++)
                for (int j = 0; j < 6; j++) {
                    K[(6 * a + i) * 6 * NN + 6 * b + j] = t[i][j];
                    K[(6 * a + 3 + i) * 6 * NN + 6 * b + j] = u[i][j];
                }
        }
    return true;
}

template <bool AVGK>
static bool layered_triangle(const ElemIn<3> &in, const fsl::ElemIn<3> &il, const MatConst &mc, const fsl::MatConst &ml,
                             const GroupConst &gc, const fsl::GroupConst &gl, double *K, double *dfixed, double *ddouble)
{
    constexpr int NR = 6 + T3Rows<AVGK>::NS;
    double compact[LayeredRows<3, NR>::SIZE], rows[(NR + 3) * 18], F[324];
    long double wide[(NR + 3) * 18];
    t3_rows<double, true, AVGK, true>(in, mc, &gc, compact, 18);
    t3_rows<double, true, AVGK>(in, mc, &gc, rows, 18);
    fsl::t3_rows<long double, true, AVGK>(il, ml, &gl, wide, 18);
    if (!layered_blocks<3, NR>(compact, 0, F)) return false;
    compare(18, NR + 3, F, rows, wide, K, dfixed, ddouble);
    return true;
}

extern "C" {

// layered elements (nen 3 or 4; avgk for triangles) of one layup
int stretched_layered(int nen, int avgk, int64_t n, const double *X, const double *nrm, const fs_layup_group *group,
                      const fs_shell_params *p, double *K, double *dfixed, double *ddouble)
{
    MatConst mc;
    fsl::MatConst ml;
    GroupConst gc;
    fsl::GroupConst gl;
    if (constants(*p, mc, ml) || prepare_group(*group, gc)) return 1;
    memset(&gl, 0, sizeof gl);
    for (int i = 0; i < 21; i++) gl.L6[i] = gc.L6[i];
    for (int i = 0; i < 3; i++) gl.LH[i] = gc.LH[i];
    for (int i = 0; i < 9; i++) gl.csmat[i] = gc.csmat[i];
    gl.thickness = gc.thickness;
    ml.drill_scale6 = mc.drill_scale6;
    for (int64_t e = 0; e < n; e++) {
        if (nen == 3) {
            const ElemIn<3> in = element<ElemIn<3>>(X + 9 * e, nrm + 9 * e, 0.0);
            const fsl::ElemIn<3> il = element<fsl::ElemIn<3>>(X + 9 * e, nrm + 9 * e, 0.0);
            const int64_t at = 324 * e;
            if (!(avgk ? layered_triangle<true> : layered_triangle<false>)(in, il, mc, ml, gc, gl, K + at, dfixed + at, ddouble + at))
                return 2;
            continue;
        }
        const ElemIn<4> in = element<ElemIn<4>, 4>(X + 12 * e, nrm + 12 * e, 0.0);
        const fsl::ElemIn<4> il = element<fsl::ElemIn<4>, 4>(X + 12 * e, nrm + 12 * e, 0.0);
        Q4Elem qe;
        fsl::Q4Elem ql;
        q4_prepare(in, gc.thickness, mc.stab_c, qe);
        fsl::q4_prepare(il, gl.thickness, ml.stab_c, ql);
        double rows[36 * 24], compact[LayeredRows<4, 32>::SIZE], F[576], td[4] = {0, 0, 0, 0}, tp[4];
        long double wide[36 * 24], tl[4] = {0, 0, 0, 0}, tq[4];
        for (int j = 0; j < 4; j++) {
            q4_point_rows<double, true>(in, qe, j, mc, &gc, rows + j * 8 * 24, 24, tp);
            for (int k = 0; k < 4; k++) td[k] += tp[k];
            fsl::q4_point_rows<long double, true>(il, ql, j, ml, &gl, wide + j * 8 * 24, 24, tq);
            for (int k = 0; k < 4; k++) tl[k] += tq[k];
        }
        q4_drill_rows<double>(in, td, mc.drill_scale, rows + 32 * 24, 24);
        fsl::q4_drill_rows<long double>(il, tl, ml.drill_scale, wide + 32 * 24, 24);
        memcpy(compact, rows, sizeof(double) * 32 * 24);
        for (int k = 0; k < 12; k++) compact[32 * 24 + k] = rows[(32 + k / 3) * 24 + 6 * (k / 3) + 3 + k % 3];
        if (!layered_blocks<4, 32>(compact, 1, F)) return 3;
        compare(24, 36, F, rows, wide, K + 576 * e, dfixed + 576 * e, ddouble + 576 * e);
    }
    return 0;
}

}  // extern "C"
