// FP64 Q1 geometry: shape functions, the multilinear map, its Jacobian and
// inverse (deal.II FE_Q<dim>(1) and MappingQ1, used by the reference at
// src/pfem2particlehandler.cpp:91,97,131,155,193,394,400,425,463 and
// src/pfem2particle.cpp:190).
//
// The FP64 form compiles this header with --fmad=false: every product and sum
// is rounded separately in the written order, the same arithmetic as an
// FMA-free CPU build, so the FP64 particle path reproduces its CPU
// restatement bit for bit.  The FP32 form reuses it (with contraction) only
// for particles that cross a cell face.
#pragma once

#include "common.cuh"

namespace pfem2 {

__device__ __forceinline__ double lag64(int b, double t) { return b ? t : 1.0 - t; }

// N_i = prod_d (b_d ? xi_d : 1 - xi_d), vertex bits b_d = (i >> d) & 1.
template <int DIM>
__device__ __forceinline__ void shape64(const double* xi, double* N)
{
#pragma unroll
    for (int i = 0; i < (1 << DIM); ++i) {
        double n = lag64(i & 1, xi[0]);
        if (DIM > 1) n = n * lag64((i >> 1) & 1, xi[1]);
        if (DIM > 2) n = n * lag64((i >> 2) & 1, xi[2]);
        N[i] = n;
    }
}

// dN_i/dxi_k = (b_k ? 1 : -1) prod_{m != k} (b_m ? xi_m : 1 - xi_m), product in m order.
template <int DIM>
__device__ __forceinline__ void shape_grad64(const double* xi, double (*G)[DIM])
{
#pragma unroll
    for (int i = 0; i < (1 << DIM); ++i)
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            double g = ((i >> k) & 1) ? 1.0 : -1.0;
#pragma unroll
            for (int m = 0; m < DIM; ++m)
                if (m != k) g = g * lag64((i >> m) & 1, xi[m]);
            G[i][k] = g;
        }
}

// The sums of products here start with their first product, as a rounded one
// that is never contracted into the next: what a start from zero gives, a
// zero's sign in sums of nothing but zeros apart (coordinates of -0.0).  18
// FP64 additions less in each Newton iteration (advect of the 37^3 cube's
// 6.3 M particles 1938 -> 1862 us).
template <int DIM>
__device__ __forceinline__ void fwd64(const double (*X)[DIM], const double* xi, double* x)
{
    double N[1 << DIM];
    shape64<DIM>(xi, N);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        double acc = __dmul_rn(N[0], X[0][d]);
#pragma unroll
        for (int i = 1; i < (1 << DIM); ++i) acc = acc + N[i] * X[i][d];
        x[d] = acc;
    }
}

template <int DIM>
__device__ __forceinline__ void jac64(const double (*X)[DIM], const double* xi, double (*J)[DIM])
{
    double G[1 << DIM][DIM];
#pragma unroll
    for (int i = 0; i < (1 << DIM); ++i)
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            double g = ((i >> k) & 1) ? 1.0 : -1.0;
#pragma unroll
            for (int m = 0; m < DIM; ++m)
                if (m != k) g = g * lag64((i >> m) & 1, xi[m]);
            G[i][k] = g;
        }
#pragma unroll
    for (int d = 0; d < DIM; ++d)
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            double acc = __dmul_rn(G[0][k], X[0][d]);
#pragma unroll
            for (int i = 1; i < (1 << DIM); ++i) acc = acc + G[i][k] * X[i][d];
            J[d][k] = acc;
        }
}

// Adjugate times reciprocal determinant; returns the determinant.
template <int DIM>
__device__ __forceinline__ double invert64(const double (*A)[DIM], double (*Ai)[DIM])
{
    if constexpr (DIM == 2) {
        const double det = A[0][0] * A[1][1] - A[0][1] * A[1][0];
        const double r = 1.0 / det;
        Ai[0][0] = A[1][1] * r;
        Ai[0][1] = -A[0][1] * r;
        Ai[1][0] = -A[1][0] * r;
        Ai[1][1] = A[0][0] * r;
        return det;
    } else {
        const double c00 = A[1][1] * A[2][2] - A[1][2] * A[2][1];
        const double c01 = A[1][2] * A[2][0] - A[1][0] * A[2][2];
        const double c02 = A[1][0] * A[2][1] - A[1][1] * A[2][0];
        const double det = A[0][0] * c00 + A[0][1] * c01 + A[0][2] * c02;
        const double r = 1.0 / det;
        Ai[0][0] = c00 * r;
        Ai[1][0] = c01 * r;
        Ai[2][0] = c02 * r;
        Ai[0][1] = (A[0][2] * A[2][1] - A[0][1] * A[2][2]) * r;
        Ai[1][1] = (A[0][0] * A[2][2] - A[0][2] * A[2][0]) * r;
        Ai[2][1] = (A[0][1] * A[2][0] - A[0][0] * A[2][1]) * r;
        Ai[0][2] = (A[0][1] * A[1][2] - A[0][2] * A[1][1]) * r;
        Ai[1][2] = (A[0][2] * A[1][0] - A[0][0] * A[1][2]) * r;
        Ai[2][2] = (A[0][0] * A[1][1] - A[0][1] * A[1][0]) * r;
        return det;
    }
}

template <int DIM>
__device__ __forceinline__ void matvec64(const double (*A)[DIM], const double* x, double* y)
{
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
        double acc = __dmul_rn(A[k][0], x[0]);
#pragma unroll
        for (int d = 1; d < DIM; ++d) acc = acc + A[k][d] * x[d];
        y[k] = acc;
    }
}

template <int DIM>
__device__ __forceinline__ double norm2_64(const double* a)
{
    double s = __dmul_rn(a[0], a[0]);
#pragma unroll
    for (int d = 1; d < DIM; ++d) s = s + a[d] * a[d];
    return s;
}

// GeometryInfo<dim>::is_inside_unit_cell(p), no tolerance; NaN is outside.
template <int DIM, typename R>
__device__ __forceinline__ bool inside_unit(const R* xi)
{
    bool in = true;
#pragma unroll
    for (int d = 0; d < DIM; ++d) in = in && (xi[d] >= R(0) && xi[d] <= R(1));
    return in;
}

template <int DIM>
__device__ __forceinline__ bool inside_unit_eps(const double* xi, double eps)
{
    bool in = true;
#pragma unroll
    for (int d = 0; d < DIM; ++d) in = in && (xi[d] >= -eps && xi[d] <= 1.0 + eps);
    return in;
}

template <int DIM>
__device__ __forceinline__ bool near_face64(const double* xi)
{
    bool nf = false;
#pragma unroll
    for (int d = 0; d < DIM; ++d) nf = nf || fabs(xi[d]) < 1e-12 || fabs(1.0 - xi[d]) < 1e-12;
    return nf;
}

// The same two tests (3D), most points decided by integer compares of the
// high words: below that of 1.0 a double is in [0, 1), between those of
// 1e-12 and the last one below 1.0 it is near neither face.
__device__ __forceinline__ bool inside_fast64(const double* xi)
{
    const bool sure = (unsigned)__double2hiint(xi[0]) < 0x3FF00000u && (unsigned)__double2hiint(xi[1]) < 0x3FF00000u &&
                      (unsigned)__double2hiint(xi[2]) < 0x3FF00000u;
    return sure || inside_unit<3>(xi);
}
__device__ __forceinline__ bool near_face_fast64(const double* xi)
{
    bool maybe = false;
#pragma unroll
    for (int d = 0; d < 3; ++d)
        maybe = maybe || (unsigned)__double2hiint(xi[d]) - 0x3D71979Au >= 0x3FEFFFFFu - 0x3D71979Au;
    return maybe && near_face64<3>(xi);
}

// 2D closed-form bilinear inverse: r = xi e + eta f + xi eta g with
// e = X1-X0, f = X2-X0, g = X3-X1-X2+X0, r = p-X0; eliminating xi leaves
// cross(f,g) eta^2 + (cross(f,e) - cross(r,g)) eta - cross(r,e) = 0, solved
// without cancellation, root nearest 1/2, xi by projection.  0 = success.
__device__ __forceinline__ int bilinear_exact64(const double (*X)[2], const double* p, double* xi)
{
    const double ex = X[1][0] - X[0][0], ey = X[1][1] - X[0][1];
    const double fx = X[2][0] - X[0][0], fy = X[2][1] - X[0][1];
    const double gx = ((X[3][0] - X[1][0]) - X[2][0]) + X[0][0];
    const double gy = ((X[3][1] - X[1][1]) - X[2][1]) + X[0][1];
    const double rx = p[0] - X[0][0], ry = p[1] - X[0][1];
    const double qa = fx * gy - fy * gx;
    const double qb = (fx * ey - fy * ex) - (rx * gy - ry * gx);
    const double qc = -(rx * ey - ry * ex);
    double eta;
    if (qa == 0.0) {
        if (qb == 0.0) return 1;
        eta = -qc / qb;
    } else {
        const double disc = qb * qb - 4.0 * qa * qc;
        if (!(disc >= 0.0)) return 1;
        const double sq = sqrt(disc);
        const double q = -0.5 * (qb + (qb >= 0.0 ? sq : -sq));
        if (q == 0.0) {
            eta = 0.0;
        } else {
            const double e1 = q / qa;
            const double e2 = qc / q;
            eta = (fabs(e1 - 0.5) < fabs(e2 - 0.5)) ? e1 : e2;
        }
    }
    const double wx = ex + eta * gx, wy = ey + eta * gy;
    const double tx = rx - eta * fx, ty = ry - eta * fy;
    const double ww = wx * wx + wy * wy;
    if (!(ww > 0.0)) return 1;
    xi[0] = (tx * wx + ty * wy) / ww;
    xi[1] = eta;
    return 0;
}

// Inverse of the least-squares affine approximation of one cell's map:
// column k of A is the mean edge vector in direction k, b = centroid - A/2.
// Written as aff = [A^-1 row-major | b]; NaN marks a singular cell.
template <int DIM>
__device__ __forceinline__ void affine_setup64(const double (*X)[DIM], double* aff)
{
    constexpr int NV = 1 << DIM;
    const double half = (double)(NV / 2);
    double A[DIM][DIM], Ai[DIM][DIM], b[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        double mean = 0.0;
#pragma unroll
        for (int i = 0; i < NV; ++i) mean = mean + X[i][d];
        mean = mean / (double)NV;
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            double sp = 0.0, sm = 0.0;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                if ((i >> k) & 1) sp = sp + X[i][d];
                else sm = sm + X[i][d];
            }
            A[d][k] = (sp - sm) / half;
        }
        double ac = 0.0;
#pragma unroll
        for (int k = 0; k < DIM; ++k) ac = ac + A[d][k] * 0.5;
        b[d] = mean - ac;
    }
    const double det = invert64<DIM>(A, Ai);
    const bool bad = !(det != 0.0) || !isfinite(det);
#pragma unroll
    for (int k = 0; k < DIM; ++k)
#pragma unroll
        for (int d = 0; d < DIM; ++d) aff[k * DIM + d] = bad ? __longlong_as_double(0x7ff8000000000000ll) : Ai[k][d];
#pragma unroll
    for (int d = 0; d < DIM; ++d) aff[DIM * DIM + d] = b[d];
}

// A row of N doubles (N even, the row 16-byte aligned) in 16-byte loads: a
// relocation's lanes read rows of different cells, and every load is a
// request per lane whatever its width.
template <int N>
__device__ __forceinline__ void load_row64(const double* __restrict__ p, double* b)
{
#pragma unroll
    for (int j = 0; j < N; j += 2) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(p + j));
        b[j] = t.x;
        b[j + 1] = t.y;
    }
}

// The N ids (4 or 8) of one cell's row.
template <int N>
__device__ __forceinline__ void load_ids(const int32_t* __restrict__ p, int32_t* id)
{
#pragma unroll
    for (int j = 0; j < N; j += 4) {
        const int4 t = __ldg(reinterpret_cast<const int4*>(p + j));
        id[j] = t.x;
        id[j + 1] = t.y;
        id[j + 2] = t.z;
        id[j + 3] = t.w;
    }
}

// Is a quad's inverse map of points within a quarter cell of it decided by its
// closed form?  With A the affine part of F and g the twist vector, F(xi) =
// centre + A (xi - 1/2) + (xi_0 - 1/2)(xi_1 - 1/2) g.  For kappa = |A^-1 g|_1
// <= 1/10 and det A > 0 the other root of the closed form's quadratic lies
// some 1 / kappa cells away, so the one it takes is the only solution near
// the cell, well conditioned; Newton from the clamped affine guess g0 (at
// most 0.45 away) satisfies Kantorovich's condition (1.2 x 0.6 x 0.15 < 1/2),
// takes full steps and keeps det J > 0; and its end test, |J^-1 (F - p)| <=
// 1e-11, passes as long as the rounding of F, 13.5 u xm, stays below that:
// xm |A^-1| <= 1600 leaves a factor of 3.  The closed form is then within
// 1e-9 of the solution, the limits of its use (1e-6) are far from that.
__device__ __forceinline__ bool mild_quad64(const double (*X)[2], const double* aff)
{
    const double gx = ((X[3][0] - X[1][0]) - X[2][0]) + X[0][0], gy = ((X[3][1] - X[1][1]) - X[2][1]) + X[0][1];
    double xm = 0.0;
    for (int i = 0; i < 4; ++i) xm = fmax(xm, fmax(fabs(X[i][0]), fabs(X[i][1])));
    const double kappa = fabs(aff[0] * gx + aff[1] * gy) + fabs(aff[2] * gx + aff[3] * gy);
    const double na = fmax(fabs(aff[0]) + fabs(aff[1]), fabs(aff[2]) + fabs(aff[3]));
    return kappa <= 0.1 && xm * na <= 1600.0 && aff[0] * aff[3] - aff[1] * aff[2] > 0.0;
}

// MappingQ1::transform_real_to_unit_cell restated (deal.II's published
// strategy): 2D closed form accepted inside the unit cell within 1e-12;
// otherwise Newton from the affine guess clamped to the unit cell, residual
// weighted by J^-1, converged below 1e-11, step halved down to 0.05 while the
// weighted residual does not drop, one restart from the clamped iterate, fail
// on det <= 0 or after 20 iterations.  0 = success.
//
// mild (2D, mild_quad64): where the closed form puts the point outside the
// cell by more than 1e-6 and less than a quarter of it, Newton would converge
// to that same point; it is returned at once.  Every particle that leaves
// its quad, and every candidate cell that does not hold it, comes here: the
// Newton iterations (two thirds of a warp's FP64 operations where one lane
// in five crosses a face) only told that the point is outside.  Turek mesh,
// 1.9 M particles, 412 k crossings a step: advect of the FP64 form 201 -> 149
// us, relocation of the FP32 form 83 -> 76, of the FP64 form 99 -> 93.
template <int DIM>
__device__ __forceinline__ int inverse_map64(const double (*X)[DIM], const double* __restrict__ aff,
                                             const double* p, double* xi_out, bool mild = false)
{
    double xi[DIM], f[DIM], x[DIM], r[DIM];
    if constexpr (DIM == 2) {
        double e[2];
        if (bilinear_exact64(X, p, e) == 0) {
            if (inside_unit_eps<2>(e, 1e-12)) {
                xi_out[0] = e[0];
                xi_out[1] = e[1];
                return 0;
            }
            const bool near = e[0] >= -0.25 && e[0] <= 1.25 && e[1] >= -0.25 && e[1] <= 1.25;
            if (mild && near && !inside_unit_eps<2>(e, 1e-6)) {
                xi_out[0] = e[0];
                xi_out[1] = e[1];
                return 0;
            }
        }
    }
    {
        double Ai[DIM][DIM], row[DIM * DIM + DIM];
        load_row64<DIM * DIM + DIM>(aff, row);
#pragma unroll
        for (int k = 0; k < DIM; ++k)
#pragma unroll
            for (int d = 0; d < DIM; ++d) Ai[k][d] = row[k * DIM + d];
        if (Ai[0][0] != Ai[0][0]) return 1;
#pragma unroll
        for (int d = 0; d < DIM; ++d) r[d] = p[d] - row[DIM * DIM + d];
        matvec64<DIM>(Ai, r, xi);
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d) xi[d] = 0.0 + xi[d];  // never -0: the Newton updates keep that
#pragma unroll
    for (int d = 0; d < DIM; ++d) xi[d] = xi[d] < 0.0 ? 0.0 : (xi[d] > 1.0 ? 1.0 : xi[d]);
    fwd64<DIM>(X, xi, x);
#pragma unroll
    for (int d = 0; d < DIM; ++d) f[d] = x[d] - p[d];
    bool restarted = false;
    for (int it = 0; it < 20; ++it) {
        double J[DIM][DIM], Ji[DIM][DIM], delta[DIM], trial[DIM], ft[DIM], dt[DIM];
        jac64<DIM>(X, xi, J);
        const double det = invert64<DIM>(J, Ji);
        if (!(det > 0.0)) return 1;
        matvec64<DIM>(Ji, f, delta);
        const double dn = norm2_64<DIM>(delta);
        if (dn <= 1e-22) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) xi_out[d] = xi[d];
            return 0;
        }
        double step = 1.0, tn = 0.0;
        bool accepted = false;
        for (int ls = 0; ls < 8; ++ls) {  // 1, 1/2, ..., 1/32 then stop
#pragma unroll
            for (int d = 0; d < DIM; ++d) trial[d] = xi[d] - step * delta[d];
            fwd64<DIM>(X, trial, x);
#pragma unroll
            for (int d = 0; d < DIM; ++d) ft[d] = x[d] - p[d];
            matvec64<DIM>(Ji, ft, dt);
            tn = norm2_64<DIM>(dt);
            if (tn < dn) {
                accepted = true;
                break;
            }
            if (step > 0.05) step = step * 0.5;
            else break;
        }
        if (!accepted) {
            if (restarted) return 1;
            restarted = true;
#pragma unroll
            for (int d = 0; d < DIM; ++d) xi[d] = xi[d] < 0.0 ? 0.0 : (xi[d] > 1.0 ? 1.0 : xi[d]);
            fwd64<DIM>(X, xi, x);
#pragma unroll
            for (int d = 0; d < DIM; ++d) f[d] = x[d] - p[d];
            continue;
        }
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            xi[d] = trial[d];
            f[d] = ft[d];
        }
        if (tn <= 1e-22) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) xi_out[d] = xi[d];
            return 0;
        }
    }
    return 1;
}

// Inverse of an affine cell's map from its stored inverse (aff = [A^-1 | b],
// x = A xi + b exactly for a parallelepiped).  0 = success (1: singular cell).
template <int DIM>
__device__ __forceinline__ int inverse_affine64(const double* __restrict__ aff, const double* p, double* xi)
{
    double row[DIM * DIM + DIM];
    load_row64<DIM * DIM + DIM>(aff, row);
    if (row[0] != row[0]) return 1;
    double r[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) r[d] = p[d] - row[DIM * DIM + d];
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
        double acc = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) acc = acc + row[k * DIM + d] * r[d];
        xi[k] = acc;
    }
    return 0;
}

// Decides inverse_map64 of a hex from its affine guess g = A^-1 (p - b) alone
// (the same operations in the same order): 0, inside, with xi = g, the value
// inverse_map64 returns; 1, outside, where it returns a point outside the
// unit cell; 2, undecided.  Only for cells that cell_setup found safe (LIN64_MAX):
// the map is affine and all its roundings together move a point by less than
// 1e-11 / sqrt(3) in reference coordinates for points up to half a cell outside,
// so that a guess inside the cell needs no clamping and its weighted residual
// passes Newton's first test (|J^-1 f|^2 <= 1e-22), and a guess more than 1e-9
// outside leads, after clamping, to one Newton step that lands within 1e-11
// of it and stops.  What is left out is the residual F(g) - p, the Jacobian
// and its inverse: 250 of the 340 FP64 operations of a sub-step.  LIN64_MAX is
// about half of that 1e-11 / sqrt(3).  One cell beyond it leaves the whole mesh
// to Newton: the bound grows with max |x| / h, and of a duct 8 long and 1 wide
// 128x32x32 cells are within it (2.86e-12) and 136x34x34 are not (3.04e-12).
constexpr double LIN64_MAX = 3e-12;
template <typename Aff>  // aff(j): the cell's j-th affine value
__device__ __forceinline__ int locate_lin64(Aff&& aff, const double* p, double* xi)
{
    double r[3], g[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) r[d] = p[d] - aff(9 + d);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double acc = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) acc = acc + aff(k * 3 + d) * r[d];
        g[k] = acc;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) xi[d] = g[d];
    if (inside_fast64(g)) return 0;
    bool out = false, near = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        out = out || g[d] < -1e-9 || g[d] > 1.0 + 1e-9;
        near = near && (g[d] >= -0.5 && g[d] <= 1.5);
    }
    return out && near ? 1 : 2;
}

// The largest reference-coordinate error of one hex's maps where it is affine
// (the bound of locate_lin64), infinity where it is not: rounding of the
// forward map up to half a cell outside (11 roundings of sum |N| |X| <= 8 xm)
// and of b (12), times |A^-1|, and the inverses' own (about cond^2 roundings).
__device__ __forceinline__ double lin64_error(const double (*X)[3], const double* aff, bool affine)
{
    constexpr double u = 1.1102230246251565e-16;
    double xm = 0.0, na = 0.0, nA = 0.0;
    for (int i = 0; i < 8; ++i)
        for (int d = 0; d < 3; ++d) xm = fmax(xm, fabs(X[i][d]));
    for (int k = 0; k < 3; ++k) {
        double s = 0.0, t = 0.0;
        for (int d = 0; d < 3; ++d) {
            s += fabs(aff[k * 3 + d]);
            t += fabs(X[1][k] - X[0][k]) * (d == 0) + fabs(X[2][k] - X[0][k]) * (d == 1) + fabs(X[4][k] - X[0][k]) * (d == 2);
        }
        na = fmax(na, s);
        nA = fmax(nA, t);
    }
    // det A > 0, as Newton asks of the Jacobian
    double e[3][3];
    for (int d = 0; d < 3; ++d)
        for (int k = 0; k < 3; ++k) e[d][k] = X[1 << k][d] - X[0][d];
    const double det = e[0][0] * (e[1][1] * e[2][2] - e[1][2] * e[2][1]) - e[0][1] * (e[1][0] * e[2][2] - e[1][2] * e[2][0]) +
                       e[0][2] * (e[1][0] * e[2][1] - e[1][1] * e[2][0]);
    const double cond = na * nA, err = na * 100.0 * u * xm + 40.0 * u * cond * cond;
    return affine && det > 0.0 && err == err ? err : __longlong_as_double(0x7ff0000000000000ll);
}

template <int DIM>
__device__ __forceinline__ void load_cell64(const double* __restrict__ cellX, uint32_t c, double (*X)[DIM])
{
    constexpr int N = (1 << DIM) * DIM;  // 8 or 24 doubles: whole 16-byte pieces
    double b[N];
    load_row64<N>(cellX + (size_t)c * N, b);
#pragma unroll
    for (int i = 0; i < (1 << DIM); ++i)
#pragma unroll
        for (int d = 0; d < DIM; ++d) X[i][d] = b[i * DIM + d];
}

// u = sum_i N_i(xi) V[dof_i] from the staged nodal velocities (VS doubles per
// DoF), accumulated from zero in vertex order: the reference's interpolation
// (src/pfem2particlehandler.cpp:96-101).
template <int DIM>
__device__ __forceinline__ void velocity_from_dofs(const int32_t* __restrict__ cd, const double* __restrict__ Va,
                                                   uint32_t c, const double* xi, double* u)
{
    constexpr int NV = 1 << DIM, VS = Dims<DIM>::VS;
    double N[NV];
    shape64<DIM>(xi, N);
#pragma unroll
    for (int d = 0; d < DIM; ++d) u[d] = 0.0;
    int32_t dof[NV];
    load_ids<NV>(cd + (size_t)c * NV, dof);
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) {
        double v[VS];
        load_row64<VS>(Va + (size_t)dof[iv] * VS, v);
#pragma unroll
        for (int d = 0; d < DIM; ++d) u[d] = u[d] + N[iv] * v[d];
    }
}

}  // namespace pfem2
