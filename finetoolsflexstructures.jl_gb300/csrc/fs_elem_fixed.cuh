// FS_FP64 elements: geometry and strain coefficients in double, the expansion
// to the global dofs and the Gram product in fixed point (fs_fixed.cuh).
//
// The rows are those of fs_elem_math.cuh (t3_rows, q4_point_rows) in two
// steps.  First, in double, the coefficients of every row in the element frame:
// u, v of a membrane row; w, the two rotations r0, r1 along the nodal triad's
// first axes and the drilling multiplier mu of a bending or shear row, node by
// node; and the largest magnitude of each kind.  Then, in fixed point, every row
// is expanded in place: the coefficients with the element basis and the
// nodal triads, whose entries are at most one, so that no row entry exceeds its
// group by more than the expansion's own factor.  Row entries come in groups with
// an exponent each, for all rows of the element: each node's translations in the
// membrane rows along each global axis (M), those in the others (T) and its
// rotations (R), and the drilling rows.  An exponent for each axis keeps the small
// components of an element near a coordinate plane: its membrane rows along the
// normal must not disturb the much smaller bending stiffness there.  One for each
// node keeps the entries of a node with small gradients, as an elongated element
// has: an entry of K is off by a few 2^-58 of its two diagonal entries' mean.
//
// That is as near as double only while the rows of one node differ by no more than
// the five bits that 58 has beyond 53, so a triangle longer than T3_LONGEST is left
// to the double kernel.  Errors of the energies of constant strains, fixed point over
// double, in the mean of 600 random triangles, the worst of nine energies, by
// elongation (longest edge squared over twice the area): at most 1.1 up to 32, 1.4
// from 32 to 64, 2.2 from 64 to 128 (a rotation's shear energy on an axis-aligned
// plate); with one exponent for all nodes 1.7 from 4 to 8, 2.7 from 16 to 32.
// Quadrilaterals: 1.4 at most but for strongly sheared ones (1.6), and the matrix is
// nearer than double's (16 to 1: 0.4 of its error, 256 to 1: 0.002), whose own rows lose more;
// none is left.  Exponents by node cost 3 % (elements, triangles, 700 x 700: 1.53 and
// 1.58 ms, quads, 360 x 360: 1.54 and 1.59); a plate of nothing but long triangles takes
// 5.0 ms instead of 2.05 (4.8 when all was double).
#pragma once

#include "fs_elem_math.cuh"
#include "fs_fixed.cuh"

#if defined(__CUDA_ARCH__)
#define FS_UNROLL _Pragma("unroll")
#define FS_UNROLL_8 _Pragma("unroll 8")
#define FS_ROLL _Pragma("unroll 1")
#else
#define FS_UNROLL
#define FS_UNROLL_8
#define FS_ROLL
#endif

namespace fs {

// the symmetric-skew triad of a node (A10 = A01, A20 = -A02, A21 = -A12)
struct Triad {
    double a00, a01, a11, a02, a12, a22;
};
struct TriadFx {
    fx a00, a01, a11, a02, a12, a22;
};

constexpr double T3_LONGEST = 32;  // longest edge squared over twice the area

// Coefficient maxima (high words) of one element, and the exponents from them.
struct FxMax {
    uint32_t m[4] = {0, 0, 0, 0}, w[4] = {0, 0, 0, 0};  // of each node: u, v | w
    uint32_t q[4] = {0, 0, 0, 0}, g[4] = {0, 0, 0, 0};  // r0, r1 | gradients
    uint32_t r = 0, u = 0;                              // drilling rows | mu
    uint32_t e[3] = {0, 0, 0};                          // e0, e1 along each axis
    FS_HD bool usable() const
    {
        bool ok = fx_usable(r) && fx_usable(u);
        FS_UNROLL
        for (int j = 0; j < 4; j++) ok = ok && fx_usable(m[j]) && fx_usable(w[j]) && fx_usable(q[j]) && fx_usable(g[j]);
        return ok;
    }
};
// a node's groups M (without the axis'), T and R
struct FxNode {
    int m, t, q;
};
struct FxExp {
    int m[4], t[4], q[4], g[4];  // each node's groups, and gradients
    int em[3];                   // units: e0, e1 along each axis
    int r, u;                    // drilling rows, mu
    bool coupled;                // some mu is not zero
    FS_HD FxNode node(int j) const { return FxNode{m[j], t[j], q[j]}; }
};
// spare: bits kept free for the longer sums of an element with several points
FS_HD FxExp fx_exponents(const FxMax &mx, int spare)
{
    FxExp x;
    x.r = fx_group(mx.r) + spare;
    x.u = fx_group(mx.u) + spare;
    x.coupled = mx.u != 0;
    FS_UNROLL
    for (int j = 0; j < 4; j++) {
        x.m[j] = fx_group(mx.m[j]) + spare;
        x.q[j] = fx_group(mx.q[j]) + spare;
        x.g[j] = fx_group(mx.g[j]);
        // |w e2 + sum h t| stays below 1.2 of the group: |w| below a half, |h| below
        // three eighths in each component (h: u + g, the drilling coupling)
        const int w = fx_group(mx.w[j]), h = x.u + x.g[j] + 2;
        x.t[j] = (x.coupled && (h > w || mx.w[j] == 0) ? h : w) + 1;
    }
    FS_UNROLL
    for (int c = 0; c < 3; c++)
        x.em[c] = fx_exp(mx.e[c]) > -60 ? fx_exp(mx.e[c]) : -60;  // below 2^-60 of the unit: counts as that
    return x;
}

// Nodal triad (nodal_triad), the drilling multipliers m0, m1 and the rotation
// block R2 (symmetric) of build_map.
FS_HD void triad_coefs(const double e[3][3], const double n[3], bool valid, Triad &A, double &m0, double &m1,
                       double R2[3])
{
    double a0 = 0.0, a1 = 0.0;
    if (valid) {
        a0 = -dot3(e[1], n);
        a1 = dot3(e[0], n);
    }
    const double x = a0 * a0 + a1 * a1;
    if (!(x > 1.0e-24) && x == x) {
        A = Triad{1.0, 0.0, 1.0, 0.0, 0.0, 1.0};
        m0 = m1 = 0.0;
        R2[0] = R2[2] = 1.0;
        R2[1] = 0.0;
        return;
    }
    double s, c;
    sinc_cosc(x, s, c);
    const double ca0 = c * a0, ca1 = c * a1;
    A.a00 = 1.0 - ca1 * a1;
    A.a01 = ca0 * a1;
    A.a11 = 1.0 - ca0 * a0;
    A.a02 = s * a1;
    A.a12 = -(s * a0);
    A.a22 = 1.0 - c * x;
    const double inv = 1.0 / A.a22;
    m0 = A.a02 * inv;
    m1 = A.a12 * inv;
    R2[0] = A.a00 - m0 * A.a02;
    R2[1] = A.a01 - m0 * A.a12;
    R2[2] = A.a11 - m1 * A.a12;
}

FS_HD TriadFx triad_fx(const Triad &A)
{
    return TriadFx{fx_make(A.a00, 0), fx_make(A.a01, 0), fx_make(A.a11, 0),
                   fx_make(A.a02, 0), fx_make(A.a12, 0), fx_make(A.a22, 0)};
}

// t[k][c] = sum_r A[r][k] e[r][c]: the triad's axes in global components
FS_HD void triad_axes(const TriadFx &A, const fx e[3][3], fx t[3][3])
{
    FS_UNROLL
    for (int c = 0; c < 3; c++) {
        FxSum s = fx_mul(A.a00, e[0][c]);
        fx_mac(s, A.a01, e[1][c]);
        fx_mac(s, fx_neg(A.a02), e[2][c]);
        t[0][c] = fx_done(s);
        s = fx_mul(A.a01, e[0][c]);
        fx_mac(s, A.a11, e[1][c]);
        fx_mac(s, fx_neg(A.a12), e[2][c]);
        t[1][c] = fx_done(s);
        s = fx_mul(A.a02, e[0][c]);
        fx_mac(s, A.a12, e[1][c]);
        fx_mac(s, A.a22, e[2][c]);
        t[2][c] = fx_done(s);
    }
}

// One row slot of an element: a coefficient (double) before the expansion, a
// row entry (fx) after it.  The slots of FX_GROUP elements lie interleaved, slot
// by slot, so that the threads of a warp, an element each, touch contiguous
// memory.
union FxSlot {
    double d;
    fx x;
    int16_t s[4];
};
constexpr int FX_GROUP = 32;
struct FxSlots {
    FxSlot *p;
    FS_HD FxSlot &operator[](int i) const { return p[i * FX_GROUP]; }
    FS_HD FxSlots operator+(int i) const { return FxSlots{p + i * FX_GROUP}; }
};

// Membrane row in place: [u0 v0 u1 v1 ..] -> NN x 3 translations
template <int NN> FS_HD void expand_membrane(FxSlots row, const fx em[2][3], const FxExp &ex)
{
    fx u[NN], v[NN];
    FS_UNROLL
    for (int j = 0; j < NN; j++) {
        u[j] = fx_make(row[2 * j].d, ex.m[j]);
        v[j] = fx_make(row[2 * j + 1].d, ex.m[j]);
    }
    FS_UNROLL
    for (int j = 0; j < NN; j++)
        FS_UNROLL
        for (int c = 0; c < 3; c++) {
            FxSum s = fx_mul(u[j], em[0][c]);
            fx_mac(s, v[j], em[1][c]);
            row[3 * j + c].x = fx_done(s);
        }
}

// Bending or shear row in place: [w0.. | r0 r1 per node | mu0..] -> NN x 6
// (translations, rotations).  g: the basis gradients (exponents ex.g).
template <int NN>
FS_HD void expand_bending(FxSlots row, bool has_w, const fx e2[3], const fx t[NN][3][3], const TriadFx A[NN],
                          const fx g[NN][2], const FxExp &ex)
{
    fx r0[NN], r1[NN], w[NN], h[NN][3];
    FS_UNROLL
    for (int j = 0; j < NN; j++) {
        w[j] = fx{0, 0};
        if (has_w) w[j] = fx_make(row[j].d, ex.t[j]);
        r0[j] = fx_make(row[NN + 2 * j].d, ex.q[j]);
        r1[j] = fx_make(row[NN + 2 * j + 1].d, ex.q[j]);
    }
    if (ex.coupled) {
        // P_r = sum_i mu_i A_i[r][:], h_j = (g_jx P_1 - g_jy P_0) / 2
        fx P[2][3], mu[NN];
        FS_UNROLL
        for (int i = 0; i < NN; i++) mu[i] = fx_make(row[3 * NN + i].d, ex.u);
        FxSum s[2][3];
        FS_UNROLL
        for (int i = 0; i < NN; i++) {
            const fx a0[3] = {A[i].a00, A[i].a01, A[i].a02}, a1[3] = {A[i].a01, A[i].a11, A[i].a12};
            FS_UNROLL
            for (int k = 0; k < 3; k++) {
                if (i == 0) {
                    s[0][k] = fx_mul(mu[i], a0[k]);
                    s[1][k] = fx_mul(mu[i], a1[k]);
                } else {
                    fx_mac(s[0][k], mu[i], a0[k]);
                    fx_mac(s[1][k], mu[i], a1[k]);
                }
            }
        }
        FS_UNROLL
        for (int k = 0; k < 3; k++) {
            P[0][k] = fx_done(s[0][k]);
            P[1][k] = fx_done(s[1][k]);
        }
        FS_UNROLL
        for (int j = 0; j < NN; j++) {
            const int sh = ex.t[j] - (ex.u + ex.g[j]) + 1;  // to the group's exponent, and the half
            FS_UNROLL
            for (int k = 0; k < 3; k++) {
                FxSum q = fx_mul(g[j][0], P[1][k]);
                fx_mac(q, fx_neg(g[j][1]), P[0][k]);
                h[j][k] = fx_split(fx_shift(fx_round(q), sh));
            }
        }
    }
    FS_UNROLL
    for (int j = 0; j < NN; j++)
        FS_UNROLL
        for (int c = 0; c < 3; c++) {
            FxSum s{0, 0};
            if (has_w) s = fx_mul(w[j], e2[c]);
            if (ex.coupled)
                FS_UNROLL
                for (int k = 0; k < 3; k++) fx_mac(s, h[j][k], t[j][k][c]);
            row[6 * j + c].x = fx_done(s);
            s = fx_mul(r0[j], t[j][0][c]);
            fx_mac(s, r1[j], t[j][1][c]);
            row[6 * j + 3 + c].x = fx_done(s);
        }
}

// What the expansion of an element (or Gauss point) needs beside its slots.
template <int NN> struct FxGeom {
    double e[3][3];    // element basis
    Triad A[NN];
    double g[NN][2];   // basis gradients
};
// maxima of the basis components and gradients
template <int NN> FS_HD void fx_max_basis(FxMax &mx, const FxGeom<NN> &geo)
{
    FS_UNROLL
    for (int j = 0; j < NN; j++) {
        fx_max(mx.g[j], geo.g[j][0]);
        fx_max(mx.g[j], geo.g[j][1]);
    }
    FS_UNROLL
    for (int c = 0; c < 3; c++) {
        fx_max(mx.e[c], geo.e[0][c]);
        fx_max(mx.e[c], geo.e[1][c]);
    }
}

// sqrt(n) and its reciprocal, each with one Newton step beyond rsqrt, and a vector
// over its length with one residual correction (as bm_quotient's; Markstein, IBM J.
// Res. Dev. 34 (1990) 111): every entry of a triangle has them as factors.  Distance of the element matrices from those in 113 bits,
// 2-norm, plates of 20 to 150 squares a side: 3.2e-16; 3.8e-16 without the
// corrections of the vectors, 4.5e-16 without either; the double kernels' 3.3e-16
FS_HD void root(double n, double &len, double &inv)
{
    const double y = rsqrt_d(n), h = n * y, hl = fma(n, y, -h);
    len = fma(0.5 * y, fma(-h, h, n), h);
    inv = fma(0.5 * y, fma(-hl, y, fma(-h, y, 1.0)), y);
}
FS_HD void unit_vector(const double v[3], double e[3], double &len, double &inv)
{
    root(dot3(v, v), len, inv);
    FS_UNROLL
    for (int c = 0; c < 3; c++) {
        const double q = v[c] * inv;
        e[c] = fma(fma(-len, q, v[c]), inv, q);
    }
}

// T3FF, homogeneous, average B: coefficients into the slots (CompactRows<3, 2>
// layout).  In the element frame the first edge lies on x: with A, C, D its
// length and the third node's coordinates, the averaged DSG shear rows
// (_add_Bsmat_o! over the three node orderings) have the closed form below in
// q = C/A, r = D/A, s = A/D.  Returns whether the triangle is longer than T3_LONGEST
// (STOP: at once, with nothing but that).
template <bool STOP = false>
FS_HD bool t3_coefs(const ElemIn<3> &in, const MatConst &mc, FxSlots slot, FxGeom<3> &geo, FxMax &mx)
{
    typedef CompactRows<3, 2> L;
    double J0[3], J1[3], (&e)[3][3] = geo.e;
    FS_UNROLL
    for (int c = 0; c < 3; c++) {
        J0[c] = in.X[1][c] - in.X[0][c];
        J1[c] = in.X[2][c] - in.X[0][c];
    }
    double a, ia, d, id;
    unit_vector(J0, e[0], a, ia);
    double w[3];
    cross3(e[0], J1, w);
    unit_vector(w, e[2], d, id);
    cross3(e[2], e[0], e[1]);
    const double q = dot3(J1, e[0]) * ia, r = d * ia, s = a * id;
    const double Jd = a * d, t = in.t;
    const double far = fmax(fabs(q), fabs(q - 1.0)) * a;
    const bool elongated = fmax(a * a, fma(far, far, d * d)) > T3_LONGEST * Jd;
    if (STOP && elongated) return true;
    const double gx0 = -ia, gx1 = ia, gy0 = (q - 1.0) * id, gy1 = -(q * id), gy2 = id;
    geo.g[0][0] = gx0; geo.g[0][1] = gy0;
    geo.g[1][0] = gx1; geo.g[1][1] = gy1;
    geo.g[2][0] = 0.0; geo.g[2][1] = gy2;
    // weights: sqrt(t Ae), sqrt(t^3/12 Ae), sqrt(t stab Ae)
    const double sm = sqrt(t * (0.5 * Jd)), sb = sm * t * 0.28867513459481288, ws = sm * t * rsqrt_d(t * t + mc.stab_c * Jd);
    double R2[3][3], m0[3], m1[3];
    FS_UNROLL
    for (int i = 0; i < 3; i++) triad_coefs(e, in.nrm[i], in.valid[i], geo.A[i], m0[i], m1[i], R2[i]);
    double ksum = 0.0;
    // a bending or shear row's rotations tx, ty in the nodal triads
    auto rotations = [&](FxSlots row, const double (&tx)[3], const double (&ty)[3]) {
        FS_UNROLL
        for (int j = 0; j < 3; j++) {
            const double r0 = tx[j] * R2[j][0] + ty[j] * R2[j][1], r1 = tx[j] * R2[j][1] + ty[j] * R2[j][2];
            const double mu = tx[j] * m0[j] + ty[j] * m1[j];
            ksum += r0 * r0;
            ksum += r1 * r1;
            fx_max(mx.q[j], r0);
            fx_max(mx.q[j], r1);
            fx_max(mx.u, mu);
            row[3 + 2 * j].d = r0;
            row[4 + 2 * j].d = r1;
            row[9 + j].d = mu;
        }
    };
    // membrane and bending: the rows of L' (u,x  v,y  u,y + v,x)
    auto membrane_bending = [&](int k, const double (&al)[3], const double (&be)[3]) {
        const FxSlots mr = slot + L::MS * k;
        double tx[3], ty[3];
        FS_UNROLL
        for (int j = 0; j < 3; j++) {
            const double u = sm * be[j], v = sm * al[j];
            fx_max(mx.m[j], u);
            fx_max(mx.m[j], v);
            mr[2 * j].d = u;
            mr[2 * j + 1].d = v;
            tx[j] = -(sb * al[j]);
            ty[j] = sb * be[j];
        }
        rotations(slot + L::BS + L::BSS * k, tx, ty);
    };
    {
        const double c0 = mc.Lps[lp(0, 0)], c1 = mc.Lps[lp(1, 0)], c2 = mc.Lps[lp(2, 0)];
        const double al[3] = {c1 * gy0 + c2 * gx0, c1 * gy1 + c2 * gx1, c1 * gy2};
        const double be[3] = {c0 * gx0 + c2 * gy0, c0 * gx1 + c2 * gy1, c2 * gy2};
        membrane_bending(0, al, be);
    }
    {
        const double c1 = mc.Lps[lp(1, 1)], c2 = mc.Lps[lp(2, 1)];
        const double al[3] = {c1 * gy0 + c2 * gx0, c1 * gy1 + c2 * gx1, c1 * gy2};
        const double be[3] = {c2 * gy0, c2 * gy1, c2 * gy2};
        membrane_bending(1, al, be);
    }
    {
        const double c2 = mc.Lps[lp(2, 2)];
        const double al[3] = {c2 * gx0, c2 * gx1, 0.0};
        const double be[3] = {c2 * gy0, c2 * gy1, c2 * gy2};
        membrane_bending(2, al, be);
    }
    {
        const double f0 = ws * mc.Lt[lp(0, 0)], f1 = ws * mc.Lt[lp(1, 0)], f2 = ws * mc.Lt[lp(1, 1)];
        const double q6 = q * (1.0 / 6), r6 = r * (1.0 / 6), s6 = s * (1.0 / 6);
        const double y0[3] = {1.0 / 3 + q6, 0.5 - q6, 1.0 / 6};                       // g_xz: thy
        const double x1[3] = {q6 - 1.0 / 3, -(1.0 / 6) - q6, -0.5};                   // g_yz: thx
        const double y1[3] = {s6 * (1.0 - q * q), s6 * q * (q - 2.0), s6 * (2.0 * q - 1.0)};  // g_yz: thy
        FxSlots row = slot + L::BS + L::BSS * 3;
        {
            const double w[3] = {f0 * gx0 + f1 * gy0, f0 * gx1 + f1 * gy1, f1 * gy2};
            const double tx[3] = {f1 * x1[0] - f0 * r6, f1 * x1[1] + f0 * r6, f1 * x1[2]};
            const double ty[3] = {f0 * y0[0] + f1 * y1[0], f0 * y0[1] + f1 * y1[1], f0 * y0[2] + f1 * y1[2]};
            FS_UNROLL
            for (int j = 0; j < 3; j++) {
                fx_max(mx.w[j], w[j]);
                row[j].d = w[j];
            }
            rotations(row, tx, ty);
        }
        row = row + L::BSS;
        const double w[3] = {f2 * gy0, f2 * gy1, f2 * gy2};
        const double tx[3] = {f2 * x1[0], f2 * x1[1], f2 * x1[2]};
        const double ty[3] = {f2 * y1[0], f2 * y1[1], f2 * y1[2]};
        FS_UNROLL
        for (int j = 0; j < 3; j++) {
            fx_max(mx.w[j], w[j]);
            row[j].d = w[j];
        }
        rotations(row, tx, ty);
    }
    // drilling factor: the mean of the nodal-basis bending diagonals
    // (src/FEMMShellT3FFModule.jl:713-727)
    const double sk = sqrt(ksum * mc.drill_scale6);
    fx_max(mx.r, sk);
    slot[L::DR].d = sk;
    fx_max_basis(mx, geo);
    return elongated;
}

// The membrane rows (MS apart) and the bending and shear rows (from BS, BSS
// apart) of an element or Gauss point expanded in place; t: the nodal triads'
// axes.
template <int NN, int MS, int BS, int BSS>
FS_HD void expand_slots(FxSlots slot, const FxGeom<NN> &geo, const FxExp &ex, fx t[NN][3][3])
{
    fx e[3][3];
    {
        fx em[2][3];
        FS_UNROLL
        for (int c = 0; c < 3; c++) {
            em[0][c] = fx_make(geo.e[0][c], ex.em[c]);
            em[1][c] = fx_make(geo.e[1][c], ex.em[c]);
            FS_UNROLL
            for (int k = 0; k < 3; k++) e[k][c] = fx_make(geo.e[k][c], 0);
        }
        FS_ROLL
        for (int k = 0; k < 3; k++) expand_membrane<NN>(slot + MS * k, em, ex);
    }
    fx g[NN][2];
    TriadFx A[NN];
    FS_UNROLL
    for (int i = 0; i < NN; i++) {
        A[i] = triad_fx(geo.A[i]);
        triad_axes(A[i], e, t[i]);
        g[i][0] = fx_make(geo.g[i][0], ex.g[i]);
        g[i][1] = fx_make(geo.g[i][1], ex.g[i]);
    }
    FS_ROLL
    for (int k = 0; k < 5; k++) expand_bending<NN>(slot + BS + BSS * k, k >= 3, e[2], t, A, g, ex);
}

// the slots of t3_coefs expanded in place, and the drilling rows
FS_HD void t3_expand(FxSlots slot, const FxGeom<3> &geo, const bool valid[3], const FxExp &ex)
{
    typedef CompactRows<3, 2> L;
    fx t[3][3][3];
    expand_slots<3, L::MS, L::BS, L::BSS>(slot, geo, ex, t);
    const fx sk = fx_make(slot[L::DR].d, ex.r);
    FS_UNROLL
    for (int i = 0; i < 3; i++)
        FS_UNROLL
        for (int c = 0; c < 3; c++) {
            const FxSum s = fx_mul(sk, t[i][2][c]);
            slot[L::DR + 3 * i + c].x = valid[i] ? fx_done(s) : fx{0, 0};
        }
}

// Q4RS, homogeneous: coefficients of Gauss point j into its Q4Compact block,
// and its share of the drilling traces (src/FEMMShellQ4RSModule.jl:807-838).
// Xr: the nodes relative to the centroid; rn: 1 / |n| of the nodal normals (0
// for a zero one); ss: square root of the stabilisation factor.  In the element
// frame the first tangent lies on x, so that the MITC rows (_Bsmat) lose their
// terms in its y component.  Returns nonzero on a singular metric.
FS_HD int q4_coefs(const double Xr[4][3], const double nrm[4][3], const bool valid[4], const double rn[4], double t,
                   double ss, int j, const MatConst &mc, FxSlots slot, FxGeom<4> &geo, FxMax &mx, double trace[4])
{
    typedef Q4Compact L;
    double gp[4][2], J0[3], J1[3], (&e)[3][3] = geo.e;
    q4_dbasis_gp(j, gp);
    FS_UNROLL
    for (int c = 0; c < 3; c++) {
        J0[c] = Xr[0][c] * gp[0][0] + Xr[1][c] * gp[1][0] + Xr[2][c] * gp[2][0] + Xr[3][c] * gp[3][0];
        J1[c] = Xr[0][c] * gp[0][1] + Xr[1][c] * gp[1][1] + Xr[2][c] * gp[2][1] + Xr[3][c] * gp[3][1];
    }
    const double n0 = dot3(J0, J0), ia = rsqrt_d(n0);
    {
        const double G12 = dot3(J0, J1), G22 = dot3(J1, J1);
        if (n0 * G22 - G12 * G12 == 0.0) return 4;
    }
    FS_UNROLL
    for (int c = 0; c < 3; c++) e[0][c] = J0[c] * ia;
    cross3(e[0], J1, e[2]);
    const double n2 = dot3(e[2], e[2]), id = rsqrt_d(n2);
    FS_UNROLL
    for (int c = 0; c < 3; c++) e[2][c] *= id;
    cross3(e[2], e[0], e[1]);
    const double j11 = n0 * ia, j12 = dot3(J1, e[0]), j22 = n2 * id, q = j12 * ia;
    double x[4], y[4];
    FS_UNROLL
    for (int a = 0; a < 4; a++) {
        x[a] = dot3(Xr[a], e[0]);
        y[a] = dot3(Xr[a], e[1]);
        geo.g[a][0] = ia * gp[a][0];
        geo.g[a][1] = id * (gp[a][1] - q * gp[a][0]);
    }
    // weights: sqrt(t Jac), sqrt(t^3/12 Jac), sqrt(t stab Jac)
    const double sm = sqrt(t * (j11 * j22)), sb = sm * t * 0.28867513459481288, ws = sm * ss;
    double R2[4][3], m0[4], m1[4], tn0[4], tn1[4];
    FS_UNROLL
    for (int i = 0; i < 4; i++) {
        triad_coefs(e, nrm[i], valid[i], geo.A[i], m0[i], m1[i], R2[i]);
        // the first two triad axes along the unit normal
        const double c0 = dot3(e[0], nrm[i]) * rn[i], c1 = dot3(e[1], nrm[i]) * rn[i], c2 = dot3(e[2], nrm[i]) * rn[i];
        const Triad &A = geo.A[i];
        tn0[i] = A.a00 * c0 + A.a01 * c1 - A.a02 * c2;
        tn1[i] = A.a01 * c0 + A.a11 * c1 - A.a12 * c2;
        trace[i] = 0.0;
    }
    auto rotations = [&](FxSlots row, const double (&tx)[4], const double (&ty)[4]) {
        FS_UNROLL
        for (int i = 0; i < 4; i++) {
            const double r0 = tx[i] * R2[i][0] + ty[i] * R2[i][1], r1 = tx[i] * R2[i][1] + ty[i] * R2[i][2];
            const double mu = tx[i] * m0[i] + ty[i] * m1[i], p = r0 * tn0[i] + r1 * tn1[i];
            trace[i] += r0 * r0;
            trace[i] += r1 * r1;
            trace[i] -= p * p;
            fx_max(mx.q[i], r0);
            fx_max(mx.q[i], r1);
            fx_max(mx.u, mu);
            row[4 + 2 * i].d = r0;
            row[5 + 2 * i].d = r1;
            row[12 + i].d = mu;
        }
    };
    auto membrane_bending = [&](int k, const double (&al)[4], const double (&be)[4]) {
        const FxSlots mr = slot + L::MS * k;
        double tx[4], ty[4];
        FS_UNROLL
        for (int i = 0; i < 4; i++) {
            const double u = sm * be[i], v = sm * al[i];
            fx_max(mx.m[i], u);
            fx_max(mx.m[i], v);
            mr[2 * i].d = u;
            mr[2 * i + 1].d = v;
            tx[i] = -(sb * al[i]);
            ty[i] = sb * be[i];
        }
        rotations(slot + L::BS + L::BSS * k, tx, ty);
    };
    {
        const double c0 = mc.Lps[lp(0, 0)], c1 = mc.Lps[lp(1, 0)], c2 = mc.Lps[lp(2, 0)];
        double al[4], be[4];
        FS_UNROLL
        for (int i = 0; i < 4; i++) {
            al[i] = c1 * geo.g[i][1] + c2 * geo.g[i][0];
            be[i] = c0 * geo.g[i][0] + c2 * geo.g[i][1];
        }
        membrane_bending(0, al, be);
    }
    {
        const double c1 = mc.Lps[lp(1, 1)], c2 = mc.Lps[lp(2, 1)];
        double al[4], be[4];
        FS_UNROLL
        for (int i = 0; i < 4; i++) {
            al[i] = c1 * geo.g[i][1] + c2 * geo.g[i][0];
            be[i] = c2 * geo.g[i][1];
        }
        membrane_bending(1, al, be);
    }
    {
        const double c2 = mc.Lps[lp(2, 2)];
        double al[4], be[4];
        FS_UNROLL
        for (int i = 0; i < 4; i++) {
            al[i] = c2 * geo.g[i][0];
            be[i] = c2 * geo.g[i][1];
        }
        membrane_bending(2, al, be);
    }
    {
        // tying lengths at the mirrored point: LA along x, LB along the second
        // direction, whose unit vector is (j12, j22) / B
        const double r = j < 2 ? -Q4_GP : Q4_GP, s = (j & 1) ? Q4_GP : -Q4_GP;
        const double x01 = x[0] - x[1], x23 = x[2] - x[3], x03 = x[0] - x[3], x12 = x[1] - x[2];
        const double y01 = y[0] - y[1], y23 = y[2] - y[3], y03 = y[0] - y[3], y12 = y[1] - y[2];
        const double rp = r + 1.0, rm = r - 1.0, sp = s + 1.0, sm1 = s - 1.0;
        const double ax = x01 * sp + x23 * sm1, ay = y01 * sp + y23 * sm1;
        const double bx = x03 * rp - x12 * rm, by = y03 * rp - y12 * rm;
        const double LA = sqrt(ax * ax + ay * ay), LB2 = bx * bx + by * by, B2 = j12 * j12 + j22 * j22;
        // 1 / (32 det), the reciprocal with one Newton step: a factor of all shear entries
        // (their energies 1.7 times as far off as in double without, 1.3 with; elements,
        // quads 360 x 360: 1.59 and 1.62 ms)
        const double rd = ia * id, d32 = fma(fma(-j11 * j22, rd, 1.0), rd, rd) * 0.03125, kb = LB2 * rsqrt_d(LB2 * B2) * d32;  // LB / B / (32 det)
        const double q0 = j22 * kb, q1 = -(j12 * kb), p1 = -(LA * d32);
        const double f0 = ws * mc.Lt[lp(0, 0)], f1 = ws * mc.Lt[lp(1, 0)], f2 = ws * mc.Lt[lp(1, 1)];
        // node-wise factors of the two terms (w, thx, thy)
        const double aw[4] = {2.0 * rp, -2.0 * rm, 2.0 * rm, -2.0 * rp}, bw[4] = {-2.0 * sp, 2.0 * sp, -2.0 * sm1, 2.0 * sm1};
        const double axx[2] = {-(y03 * rp), y12 * rm}, axy[2] = {x03 * rp, -(x12 * rm)};    // nodes 0, 3 | 1, 2
        const double bxx[2] = {y01 * sp, y23 * sm1}, bxy[2] = {-(x01 * sp), -(x23 * sm1)};  // nodes 0, 1 | 2, 3
        double w1[4], x1[4], y1[4];
        FS_UNROLL
        for (int i = 0; i < 4; i++) {
            const int ka = (i == 0 || i == 3) ? 0 : 1, kq = i < 2 ? 0 : 1;
            w1[i] = p1 * aw[i] + q1 * bw[i];
            x1[i] = p1 * axx[ka] + q1 * bxx[kq];
            y1[i] = p1 * axy[ka] + q1 * bxy[kq];
        }
        const double g0 = f0 * q0;
        FxSlots row = slot + L::BS + L::BSS * 3;
        double tx[4], ty[4];
        FS_UNROLL
        for (int i = 0; i < 4; i++) {
            const int kq = i < 2 ? 0 : 1;
            const double w = g0 * bw[i] + f1 * w1[i];
            fx_max(mx.w[i], w);
            row[i].d = w;
            tx[i] = g0 * bxx[kq] + f1 * x1[i];
            ty[i] = g0 * bxy[kq] + f1 * y1[i];
        }
        rotations(row, tx, ty);
        row = row + L::BSS;
        FS_UNROLL
        for (int i = 0; i < 4; i++) {
            const double w = f2 * w1[i];
            fx_max(mx.w[i], w);
            row[i].d = w;
            tx[i] = f2 * x1[i];
            ty[i] = f2 * y1[i];
        }
        rotations(row, tx, ty);
    }
    fx_max_basis(mx, geo);
    return 0;
}

// 3 x 3 sums of products, and the pieces of a node block from them
struct FxSums {
    int64_t hh[3][3], c[3][3];
    FS_HD void zero()
    {
        FS_UNROLL
        for (int i = 0; i < 3; i++)
            FS_UNROLL
            for (int j = 0; j < 3; j++) hh[i][j] = c[i][j] = 0;
    }
    // entries (i, j), j >= i only on a diagonal block (UPPER)
    template <bool UPPER> FS_HD void add(const fx (&a)[3], const fx *b)
    {
        FS_UNROLL
        for (int i = 0; i < 3; i++)
            FS_UNROLL
            for (int j = UPPER ? i : 0; j < 3; j++) {
                hh[i][j] += (int64_t)a[i].h * b[j].h;
                c[i][j] += (int64_t)a[i].h * b[j].l;
                c[i][j] += (int64_t)a[i].l * b[j].h;
            }
    }
    FS_HD double value(int i, int j, int E) const { return fx_double(FxSum{hh[i][j], c[i][j]}, E); }
};
template <int N> FS_HD void fx_load(FxSlots p, fx (&v)[N])
{
    FS_UNROLL
    for (int i = 0; i < N; i++) v[i] = p[i].x;
}

// One node block (p, q) of K from expanded rows: NP row sets (Gauss points),
// `step` apart, of 3 membrane rows (MS apart, 3 values a node) and 5 bending and
// shear rows (from BS, BSS apart, 6 values a node), and the node's drilling row
// on a diagonal block.  top: rows 0..2 of the block into o, bottom: rows 3..5 (on a
// diagonal block without its first three columns, the transpose of the top's
// last three).
// ex: the exponents, an FxExp or where they lie (node(), em and r of it).
template <int NP, int MS, int BS, int BSS, bool DIAG, class X>
FS_HD void fx_block_top(FxSlots rows, int step, int p, int q, const X &ex, double o[3][6])
{
    const FxNode a = ex.node(p), b = ex.node(q);
    FxSums m, tt, tr;
    m.zero();
    FS_ROLL
    for (int pt = 0; pt < NP; pt++) {
        FS_UNROLL
        for (int k = 0; k < 3; k++) {
            fx x[3], y[3];
            fx_load(rows + pt * step + MS * k + 3 * p, x);
            fx_load(rows + pt * step + MS * k + 3 * q, y);
            m.template add<DIAG>(x, y);
        }
    }
    FS_UNROLL
    for (int i = 0; i < 3; i++)
        FS_UNROLL
        for (int j = DIAG ? i : 0; j < 3; j++) o[i][j] = m.value(i, j, ex.em[i] + ex.em[j] + a.m + b.m);
    tt.zero();
    tr.zero();
    FS_ROLL
    for (int pt = 0; pt < NP; pt++) {
        FS_UNROLL
        for (int k = 0; k < 5; k++) {
            fx x[3], y[6];
            fx_load(rows + pt * step + BS + BSS * k + 6 * p, x);
            fx_load(rows + pt * step + BS + BSS * k + 6 * q, y);
            tt.template add<DIAG>(x, y);
            tr.template add<false>(x, y + 3);
        }
    }
    FS_UNROLL
    for (int i = 0; i < 3; i++) {
        FS_UNROLL
        for (int j = DIAG ? i : 0; j < 3; j++) {
            o[i][j] += tt.value(i, j, a.t + b.t);
            if (DIAG && j > i) o[j][i] = o[i][j];
        }
        FS_UNROLL
        for (int j = 0; j < 3; j++) o[i][3 + j] = tr.value(i, j, a.t + b.q);
    }
}
template <int NP, int BS, int BSS, bool DIAG, class X>
FS_HD void fx_block_bottom(FxSlots rows, int step, int p, int q, FxSlots drill, const X &ex, double o[3][6])
{
    const FxNode a = ex.node(p), b = ex.node(q);
    const int top = 2 * (a.q > ex.r ? a.q : ex.r);  // the larger of the rows' and the drilling row's products
    FxSums rt, rr, dd;
    rt.zero();
    rr.zero();
    FS_ROLL
    for (int pt = 0; pt < NP; pt++) {
        FS_UNROLL
        for (int k = 0; k < 5; k++) {
            fx x[3], y[6];
            fx_load(rows + pt * step + BS + BSS * k + 6 * p + 3, x);
            fx_load(rows + pt * step + BS + BSS * k + 6 * q, y);
            if (!DIAG) rt.template add<false>(x, y);
            rr.template add<DIAG>(x, y + 3);
        }
    }
    if (DIAG) {
        fx d[3];
        fx_load(drill, d);
        dd.zero();
        dd.template add<true>(d, d);
    }
    FS_UNROLL
    for (int i = 0; i < 3; i++) {
        if (!DIAG) {
            FS_UNROLL
            for (int j = 0; j < 3; j++) o[i][j] = rt.value(i, j, a.q + b.t);
        }
        FS_UNROLL
        for (int j = DIAG ? i : 0; j < 3; j++) {
            if (DIAG)
                o[i][3 + j] = fx_double(FxSum{fx_shift(fx_round(FxSum{rr.hh[i][j], rr.c[i][j]}), top - 2 * a.q) +
                                                  fx_shift(fx_round(FxSum{dd.hh[i][j], dd.c[i][j]}), top - 2 * ex.r), 0}, top);
            else
                o[i][3 + j] = rr.value(i, j, a.q + b.q);
            if (DIAG && j > i) o[j][3 + i] = o[i][3 + j];
        }
    }
}

// Double rows of a layered element multiplied in fixed point (FS_FP64): the
// values of each dof over all rows share an exponent, so that a row entry is kept
// to 2^-58 of its dof's largest, an entry of K to a few 2^-58 of its two diagonal
// entries' mean, and the products are exact sums of integers (fs_fixed.cuh),
// rounded once.  In double the products are half of the kernel's double operations
// (T3FFComp, 257 x 190: 0.65 ms, now 0.55; Q4RSComp, 512 x 512: 10.6 and 8.1).
typedef uint64_t DofExp;  // a node's six exponents, 10 bits each, from -512
FS_HD int dof_exp(DofExp e, int k) { return (int)((uint32_t)(e >> 10 * k) & 1023u) - 512; }
template <int NN> struct DofMax {
    uint32_t m[NN][6];
    FS_HD void zero()
    {
        FS_UNROLL
        for (int k = 0; k < 6 * NN; k++) m[k / 6][k % 6] = 0;
    }
    FS_HD void row(const double *r)
    {
        FS_UNROLL
        for (int k = 0; k < 6 * NN; k++) fx_max(m[k / 6][k % 6], r[k]);
    }
    FS_HD bool usable() const
    {
        bool ok = true;
        FS_UNROLL
        for (int k = 0; k < 6 * NN; k++) ok = ok && fx_usable(m[k / 6][k % 6]);
        return ok;
    }
    // spare: bits kept free for long sums
    FS_HD DofExp exponents(int a, int spare) const
    {
        DofExp e = 0;
        FS_UNROLL
        for (int k = 0; k < 6; k++) e |= (DofExp)(uint32_t)(fx_group(m[a][k]) + spare + 512) << 10 * k;
        return e;
    }
};
// a double replaced by its fixed-point number
FS_HD void to_fixed(double *p, int E) { *reinterpret_cast<fx *>(p) = fx_make(*p, E); }

// Rows i0 .. i0 + 2 (i0 = 0 or 3) of node block (a, b) from NR rows (stride RS) in
// fixed point; UPPER: of a diagonal block (i0 = I0), its entries (i, j), j >= i, with
// the drilling row of the node (dr: its rotations)
template <int NR, int RS, bool UPPER, int I0>
FS_HD void fixed_rows(const double *rows, const double *dr, int a, int b, DofExp Ea, DofExp Eb, double (&o)[3][6], int i0 = I0)
{
    FxSum s[3][6];
    FS_UNROLL
    for (int i = 0; i < 3; i++)
        FS_UNROLL
        for (int j = 0; j < 6; j++) s[i][j] = FxSum{0, 0};
    const fx *ra = reinterpret_cast<const fx *>(rows) + 6 * a + i0, *rb = reinterpret_cast<const fx *>(rows) + 6 * b;
    FS_UNROLL_8
    for (int r = 0; r < NR; r++) {
        fx x[3], y[6];
        FS_UNROLL
        for (int i = 0; i < 3; i++) x[i] = ra[r * RS + i];
        FS_UNROLL
        for (int j = UPPER ? I0 : 0; j < 6; j++) y[j] = rb[r * RS + j];
        FS_UNROLL
        for (int i = 0; i < 3; i++)
            FS_UNROLL
            for (int j = UPPER ? I0 + i : 0; j < 6; j++) fx_mac(s[i][j], x[i], y[j]);
    }
    if (UPPER && I0 == 3) {
        fx d[3];
        FS_UNROLL
        for (int i = 0; i < 3; i++) d[i] = reinterpret_cast<const fx *>(dr)[i];
        FS_UNROLL
        for (int i = 0; i < 3; i++)
            FS_UNROLL
            for (int j = i; j < 3; j++) fx_mac(s[i][3 + j], d[i], d[j]);
    }
    Ea >>= 10 * i0;
    FS_UNROLL
    for (int i = 0; i < 3; i++)
        FS_UNROLL
        for (int j = UPPER ? I0 + i : 0; j < 6; j++) o[i][j] = fx_double(s[i][j], dof_exp(Ea, i) + dof_exp(Eb, j));
}

}  // namespace fs
