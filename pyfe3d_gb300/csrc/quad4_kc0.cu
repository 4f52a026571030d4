// Quad4 constitutive stiffness KC0: Quad4.update_KC0 (pyfe3d/quad4.pyx:1204-1313)
// with the local matrix of _update_probe_KC0ve (pyfe3d/quad4.pyx:755-1171).
//
// GB300 organisation.  An FP64 instruction occupies the FP64 pipe for the
// whole warp whatever the number of active lanes, and FP64 issues at 1/64 of
// the FP32 rate, so the kernel counts FP64 warp-instructions per element:
//
//   phase A   one thread per element (FP64): frame R (and material cosines),
//             flatness test, constitutive matrices in the evaluation frame,
//             nodal coordinates relative to node 1, thin/thick flag.  Flat
//             isotropic elements need no frame (kc0_setup_flat_iso).
//   phase A2  one thread per (element, point) at the 4 Gauss points and the
//             centre: Jacobian and Cartesian shape derivatives, computed in
//             float-float (FP32 pipe) for flat elements.
//   phase B   16 lanes per element, one per node pair (a, b): the tensor
//             H^pq_ab = sum_points w detJ D^p N_a D^q N_b (p, q in
//             {N, d/dx, d/dy}) accumulated in float-float and converted to
//             double with integer operations, then the 6x6 block
//             K_ab = sum_pq C^pq H^pq in FP64 added onto the staged values
//             in row groups (no lane holds a whole block: for isotropic
//             sections -- rotation-invariant A, D, E and B = 0 -- the 18
//             non-zeros in two groups, otherwise three rows at a time);
//             current values that are all zeros are not added to but stored
//             over, and entries that are exact zeros are not multiplied out;
//   write-out each warp streams its two staged elements (576 values each)
//             with the coalesced += read-modify-write and the indices.
//
// CTAs of 8 warps, two per SM (128 registers): the last warp runs phase A one
// tile ahead into the other half of a double buffer, the 7 others run A2 and B
// and write out, four elements each per tile, with one barrier per tile.  (With
// phase A on a warp of the same tile the others waited for it: 20,000 of a
// tile's 70,000 cycles.)  1,000,000 flat isotropic elements with indices onto
// cleared values 3.56 -> 3.06 ms, against 2.95 ms for reading and writing the
// values and writing the indices with the same stores and no element work; DRAM
// at 6.0 TB/s.  90,000 elements into CSR 0.73 -> 0.50 ms, 28,800
// laminated elements of a cylinder 0.42 -> 0.38 ms.
//
// Flat elements whose normal is +Z (r13 = r23 = r31 = r32 = 0) are evaluated
// in the global frame with in-plane rotated constitutive matrices (no
// rotation at all for isotropic sections), which equals R Ke R^T without the
// transform.  Other elements, and the probe mode that reads the element
// state, are evaluated in FP64 in the element frame and rotated per block.
#include "fe3d_internal.h"
#include "ff.cuh"
#include "quad4_common.cuh"

namespace fe3d {
namespace {

constexpr int KCW = 7;                  // consumer warps of a CTA; one more runs phase A
constexpr int KNT = 32 * (KCW + 1);     // threads per CTA
constexpr int KPER = 4;                 // elements per consumer warp and tile at most (two per round)
constexpr int KT = KCW * KPER;          // elements per tile at most (phase A: one lane each)
constexpr int KMINB = 2;                // CTAs per SM
static_assert(KT <= 32, "phase A is one warp");
constexpr int KPTS = 5;   // 4 Gauss points + centre
constexpr int KSLOT = 9;  // per point: w detJ, Nx[4], Ny[4] (N is the same for every element)

// KF_SPLIT: (u, v, rz) and (w, rx, ry) do not couple (evaluated in the global
// frame with B = 0); KF_B0: B = 0; KF_FREE (CSR): no fixed DOF
enum : int { KF_VALID = 1, KF_THICK = 2, KF_FP64 = 4, KF_ISO = 8, KF_B0 = 16, KF_SPLIT = 32, KF_FREE = 64 };

union Slot {
    double d;
    ff f;
};

struct __align__(16) KElem {
    double R[9];
    double A[6], B[6], D[6];  // 11 12 16 22 26 66
    double ap, am;            // A66 + 1/4, A66 - 1/4: with the unit drilling weight
    double es[3];
    Slot xy[8];
    long long init_k;
    long long c[4];
    int flags;
    int pad;
};

struct KSmem {
    KElem el[2][KT];  // the tile in work, and the next one that phase A fills
    Slot gp[KT][KPTS][KSLOT];
    ff shape[KPTS][3][4];
    double stage[KCW][2][24 * KROW];
};

// shape-function values and natural derivatives at the 5 points, float-float:
// [point][0: N, 1: dN/dxi, 2: dN/deta][node]
__constant__ ff c_shape[KPTS][3][4];

// Set-up of a flat isotropic element with its normal along +z, which needs no
// frame: the decisions of q4_rotation + is_flat + iso_section, taken from the
// coordinates and the record with 20 FP64 instructions instead of about 200.
// Phase A is the serial part of a tile (one warp works, each FP64 instruction
// takes it 64 cycles), so this is what small meshes and the tile rate wait for.
// Returns false, with nothing decided, for any other element.
__device__ __forceinline__ bool kc0_setup_flat_iso(const Q4Args &a, const long long *c, const double *P, KElem &s) {
    double X[4], Y[4], Z[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const double *q = a.x + c[i] / 2;
        X[i] = q[0];
        Y[i] = q[1];
        Z[i] = q[2];
    }
    // r13 = r23 = r31 = r32 = 0: the diagonals have no z component
    bool flat = is_eq(Z[0], Z[2]) && is_eq(Z[1], Z[3]) && is_finite(Z[0]) && is_finite(Z[1]);
    double xy[8];
    bool safe = true;
    xy[0] = xy[1] = 0.;
#pragma unroll
    for (int i = 1; i < 4; i++) {
        xy[2 * i] = X[i] - X[0];
        xy[2 * i + 1] = Y[i] - Y[0];
        safe &= ff_safe(xy[2 * i]) && ff_safe(xy[2 * i + 1]);
    }
    const double vx = X[1] - X[3], vy = Y[1] - Y[3];
    flat &= is_pos(vx * xy[5] - vy * xy[4]);
    if (!flat || !safe) return false;
    const double E44 = P[SP_E44] * P[SP_SCF23];
    const double E45 = P[SP_E45] * 0.5 * (P[SP_SCF13] + P[SP_SCF23]);
    const double E55 = P[SP_E55] * P[SP_SCF13];
    const double A11 = P[SP_A11], A12 = P[SP_A12], A66 = P[SP_A66];
    const double D11 = P[SP_D11], D12 = P[SP_D12], D66 = P[SP_D66];
    bool iso = is_zero(P[SP_A16]) && is_zero(P[SP_A26]) && is_zero(P[SP_D16]) && is_zero(P[SP_D26]);
#pragma unroll
    for (int i = 0; i < 6; i++) iso &= is_zero(P[SP_B11 + i]);
    iso &= is_eq(A11, P[SP_A22]) && is_eq(D11, P[SP_D22]) && is_zero(E45) && is_eq(E44, E55);
    const double eps = 64. * 2.220446049250313e-16;
    // |x| <= y of non-negative doubles compares their bits
    iso &= dbits(fabs(A66 - 0.5 * (A11 - A12))) <= dbits(eps * fabs(A11));
    iso &= dbits(fabs(D66 - 0.5 * (D11 - D12))) <= dbits(eps * fabs(D11));
    if (!iso) return false;
    s.A[0] = A11;
    s.A[1] = A12;
    s.D[0] = D11;
    s.D[1] = D12;
    s.D[5] = D66;
    s.ap = A66 + 0.25;
    s.am = A66 - 0.25;
    s.es[0] = E44;
    s.es[1] = 0.;
    s.es[2] = E55;
    ff q[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        q[i] = i < 2 ? ff{0.f, 0.f} : ff_from_double(xy[i]);
        s.xy[i].f = q[i];
    }
    // h / sqrt(area) >= 1, in floats where they decide it
    const double h = P[SP_H];
    const float hf = (float)h;
    const float t1 = q[2].h * q[5].h, t2 = q[4].h * q[3].h, t3 = q[4].h * q[7].h, t4 = q[6].h * q[5].h;
    const float ar = 0.5f * fabsf((t1 - t2) + (t3 - t4));
    const float er = 1e-6f * (fabsf(t1) + fabsf(t2) + fabsf(t3) + fabsf(t4)), hh = hf * hf;
    bool thick = false;
    if (!(hf > 0.f && hh * 1.00001f < ar - er)) {
        if (hf > 0.f && hh > (ar + er) * 1.00001f) {
            thick = true;
        } else {
            const double sq = sqrt(shoelace(xy));
            thick = h >= sq || h / sq >= 1.;
        }
    }
    s.flags = KF_VALID | KF_ISO | KF_B0 | KF_SPLIT | (thick ? KF_THICK : 0);
    return true;
}

// Element set-up shared by the triplet and the CSR kernels: frame,
// flatness, constitutive data and nodal coordinates of element e with DOF
// offsets c[4]; ok carries the caller's own checks.
__device__ void kc0_elem_setup(const Q4Args &a, int64_t e, const long long *c, bool ok, KElem &s) {
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (c[i] < 0 || (a.x && c[i] / 2 + 3 > a.nx)) ok = false;
    const int64_t p = a.pid ? (int64_t)a.pid[e] : e;
    if (p < 0 || p >= a.nprops) ok = false;
    if (!ok) {
        raise_error(a.err, kErrBounds);
        return;
    }
    if (a.x && kc0_setup_flat_iso(a, c, a.props + (int64_t)SP_STRIDE * p, s)) return;
    const double *P = a.props + (int64_t)SP_STRIDE * p;
    double R[9], m[4] = {1., 0., 0., 1.}, xy[8], ar;
    bool fp64 = true;
    if (a.x) {
        const double *pp[4] = {a.x + c[0] / 2, a.x + c[1] / 2, a.x + c[2] / 2, a.x + c[3] / 2};
        q4_rotation(pp[0], pp[1], pp[2], pp[3], a.xmat ? a.xmat + (int64_t)a.xmat_stride * e : nullptr,
                    R, m);
        if (is_flat(R)) {
            bool safe = true;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                xy[2 * i] = pp[i][0] - pp[0][0];
                xy[2 * i + 1] = pp[i][1] - pp[0][1];
                safe &= ff_safe(xy[2 * i]) && ff_safe(xy[2 * i + 1]);
            }
            fp64 = !safe;
        }
        if (fp64) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                double q[3];
                to_local(R, pp[i], q);
                xy[2 * i] = q[0];
                xy[2 * i + 1] = q[1];
            }
        }
        q4_constitutive_packed(P, m, R, !fp64, s.A, s.B, s.D, s.es);
        ar = shoelace(xy);
    } else {
#pragma unroll
        for (int i = 0; i < 9; i++) R[i] = a.R[9 * e + i];
#pragma unroll
        for (int i = 0; i < 4; i++) m[i] = a.m[4 * e + i];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            xy[2 * i] = a.xe[12 * e + 3 * i];
            xy[2 * i + 1] = a.xe[12 * e + 3 * i + 1];
        }
        q4_constitutive_packed(P, m, R, false, s.A, s.B, s.D, s.es);
        ar = a.area[e];
    }
    s.ap = s.A[5] + 0.25;
    s.am = s.A[5] - 0.25;
    bool b0 = true;
#pragma unroll
    for (int i = 0; i < 6; i++) b0 &= is_zero(s.B[i]);
#pragma unroll
    for (int i = 0; i < 9; i++) s.R[i] = R[i];
    if (fp64) {
#pragma unroll
        for (int i = 0; i < 8; i++) s.xy[i].d = xy[i];
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) s.xy[i].f = ff_from_double(xy[i]);
    }
    // h / sqrt(area) >= 1 as the reference evaluates it; the division only
    // decides when h < sqrt(area) (h >= sqrt(area) implies the rounded
    // quotient is >= 1)
    const double sq = sqrt(ar);
    const bool thick = P[SP_H] >= sq || P[SP_H] / sq >= 1.;
    s.flags = KF_VALID | (thick ? KF_THICK : 0) | (fp64 ? KF_FP64 : 0) | (b0 ? KF_B0 : 0) |
              (b0 && !fp64 ? KF_SPLIT : 0);
}

__device__ void kc0_phase_a2(const Q4Args &a, int64_t e, KElem &s) {
    s.flags = 0;
    long long c[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        c[i] = a.cdof[4 * e + i];
        s.c[i] = c[i];
    }
    const long long k0 = a.init_k[e];
    s.init_k = k0;
    kc0_elem_setup(a, e, c, k0 >= 0 && k0 + 576 <= a.nk, s);
}

// Jacobian and Cartesian derivatives at point g in float-float.
__device__ void point_ff(const KElem &s, const ff (*shape)[3][4], int g, Slot *o) {
    ff x[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        x[i] = s.xy[2 * i].f;
        y[i] = s.xy[2 * i + 1].f;
    }
    ff J11 = ff_mul(x[0], shape[g][1][0]), J12 = ff_mul(y[0], shape[g][1][0]);
    ff J21 = ff_mul(x[0], shape[g][2][0]), J22 = ff_mul(y[0], shape[g][2][0]);
#pragma unroll
    for (int i = 1; i < 4; i++) {
        J11 = ff_fma(x[i], shape[g][1][i], J11);
        J12 = ff_fma(y[i], shape[g][1][i], J12);
        J21 = ff_fma(x[i], shape[g][2][i], J21);
        J22 = ff_fma(y[i], shape[g][2][i], J22);
    }
    const ff det = ff_fma(J11, J22, ff_neg(ff_mul(J12, J21)));
    const ff inv = ff_rcp(det);
    o[0].f = (g == 4) ? ff_scale(det, 4.f) : det;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const ff dxi = shape[g][1][i], deta = shape[g][2][i];
        o[1 + i].f = ff_mul(ff_fma(J22, dxi, ff_neg(ff_mul(J12, deta))), inv);
        o[5 + i].f = ff_mul(ff_fma(J11, deta, ff_neg(ff_mul(J21, dxi))), inv);
    }
}

__device__ __forceinline__ ff ffz() { return {0.f, 0.f}; }


// Streams one staged element (24 x KROW doubles: current values + K) to the
// caller's arrays at k0: values and, unless values_only, the indices of the
// element's DOF offsets c[4].
__device__ __forceinline__ void write_staged(const Q4Args &a, const double *sv, long long k0, const long long *c,
                                             int lane) {
    double *kv = a.Kv + k0;
    if (a.vec16 && !(k0 & 1)) {
        // 16-byte stores: slots (2 lane + 64 j, + 1) share the row and the
        // column node
        long long *kr = (long long *)a.Kr + k0, *kc = (long long *)a.Kc + k0;
        int row = lane / 12, col = 2 * lane - 24 * row;
#pragma unroll 3
        for (int j = 0; j < 9; j++) {
            const int i = 2 * lane + 64 * j;
            *reinterpret_cast<double2 *>(kv + i) = *reinterpret_cast<const double2 *>(sv + row * KROW + col);
            if (!a.values_only) {
                const int ra = row / 6, cb = col / 6;
                const long long r = c[ra] + (row - 6 * ra), c0 = c[cb] + (col - 6 * cb);
                *reinterpret_cast<longlong2 *>(kr + i) = make_longlong2(r, r);
                *reinterpret_cast<longlong2 *>(kc + i) = make_longlong2(c0, c0 + 1);
            }
            col += 16;
            row += 2;
            if (col >= 24) {
                col -= 24;
                row += 1;
            }
        }
        return;
    }
#pragma unroll 6
    for (int i = lane; i < 576; i += 32) {
        const int row = i / 24, col = i - row * 24;
        kv[i] = sv[row * KROW + col];
    }
    if (!a.values_only) {
        long long *kr = (long long *)a.Kr + k0, *kc = (long long *)a.Kc + k0;
#pragma unroll 6
        for (int i = lane; i < 576; i += 32) {
            const int row = i / 24, col = i - row * 24;
            kr[i] = c[row / 6] + row % 6;
            kc[i] = c[col / 6] + col % 6;
        }
    }
}

// N_i at point g in FP64, the expression of quad_derivs (elements evaluated
// in FP64 only).
__device__ __forceinline__ double shape_n(int g, int i) {
    double xi, eta;
    point_coords(g, xi, eta);
    const double sx = (i == 1 || i == 2) ? 1. : -1., sy = (i >= 2) ? 1. : -1.;
    return 0.25 * (1 + sx * xi) * (1 + sy * eta);
}

// The 4-point tensor H^pq_ab = sum_g w detJ D^p N_a D^q N_b (p, q in
// {N, d/dx, d/dy}) of node pair (na, nb) of element slot el: accumulated in
// float-float and rounded to double, or in FP64 for elements evaluated in
// FP64 (FF = false).  The entries (N, d) and (d, N) are halved, as the drilling
// penalty uses them.
template <bool FF>
__device__ __forceinline__ void pair_h(const KSmem &S, int el, int na, int nb, double H[3][3]) {
    if (FF) {
        ff h[3][3];
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
            for (int q = 0; q < 3; q++) h[p][q] = ffz();
        // (rolled: a quarter of the code, which the kernel otherwise fetches
        // from beyond the instruction cache: 4.27 -> 4.12 ms per 1M elements)
#pragma unroll 1
        for (int g = 0; g < 4; g++) {
            const Slot *o = S.gp[el][g];
            const ff w = o[0].f;
            const ff va[3] = {ff_mul(w, S.shape[g][0][na]), ff_mul(w, o[1 + na].f), ff_mul(w, o[5 + na].f)};
            const ff vb[3] = {S.shape[g][0][nb], o[1 + nb].f, o[5 + nb].f};
#pragma unroll
            for (int p = 0; p < 3; p++)
#pragma unroll
                for (int q = 0; q < 3; q++) h[p][q] = ff_fma(va[p], vb[q], h[p][q]);
        }
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
            for (int q = 0; q < 3; q++)
                H[p][q] = ff_to_double((p == 0) != (q == 0) ? ff_scale(h[p][q], 0.5f) : h[p][q]);
    } else {
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
            for (int q = 0; q < 3; q++) H[p][q] = 0.;
#pragma unroll
        for (int g = 0; g < 4; g++) {
            const Slot *o = S.gp[el][g];
            const double w = o[0].d;
            const double va[3] = {w * shape_n(g, na), w * o[1 + na].d, w * o[5 + na].d};
            const double vb[3] = {shape_n(g, nb), o[1 + nb].d, o[5 + nb].d};
#pragma unroll
            for (int p = 0; p < 3; p++)
#pragma unroll
                for (int q = 0; q < 3; q++) H[p][q] += va[p] * vb[q];
        }
        H[0][1] *= 0.5;
        H[0][2] *= 0.5;
        H[1][0] *= 0.5;
        H[2][0] *= 0.5;
    }
}

// The centre-point (one-point rule) tensor H0^pq_ab, entry by entry.
template <bool FF>
struct CentreH;
template <>
struct CentreH<true> {
    ff a[3], b[3];
    __device__ __forceinline__ CentreH(const KSmem &S, int el, int na, int nb) {
        const Slot *o = S.gp[el][4];
        const ff w = o[0].f;
        a[0] = ff_mul(w, S.shape[4][0][na]);
        a[1] = ff_mul(w, o[1 + na].f);
        a[2] = ff_mul(w, o[5 + na].f);
        b[0] = S.shape[4][0][nb];
        b[1] = o[1 + nb].f;
        b[2] = o[5 + nb].f;
    }
    __device__ __forceinline__ double operator()(int p, int q) const { return ff_to_double(ff_mul(a[p], b[q])); }
};
template <>
struct CentreH<false> {
    double a[3], b[3];
    __device__ __forceinline__ CentreH(const KSmem &S, int el, int na, int nb) {
        const Slot *o = S.gp[el][4];
        const double w = o[0].d;
        a[0] = w * shape_n(4, na);
        a[1] = w * o[1 + na].d;
        a[2] = w * o[5 + na].d;
        b[0] = shape_n(4, nb);
        b[1] = o[1 + nb].d;
        b[2] = o[5 + nb].d;
    }
    __device__ __forceinline__ double operator()(int p, int q) const { return a[p] * b[q]; }
};

__device__ __forceinline__ double2 *staged(double *st, int na, int nb, int m, int n) {
    return reinterpret_cast<double2 *>(st + (6 * na + m) * KROW + 6 * nb + n);
}

// Adds (x, y) onto the staged pair (row m of node na, columns n, n + 1 of node
// nb); X, Y false: that entry of the block is an exact zero and stays as it
// is.  CLEAR: the lane's staged entries are known to be zeros, so the sum is
// the entry itself.
template <bool CLEAR, bool X = true, bool Y = true>
__device__ __forceinline__ void add2(double *st, int na, int nb, int m, int n, double x, double y) {
    double2 *q = staged(st, na, nb, m, n);
    if (CLEAR && X && Y) {
        *q = make_double2(x, y);
    } else if (CLEAR) {
        if (X) q->x = x;
        if (Y) q->y = y;
    } else {
        double2 o = *q;
        if (X) o.x += x;
        if (Y) o.y += y;
        *q = o;
    }
}

// Whether the current values that the block of every lane adds to are zeros (a
// cleared array, assigned CSR blocks): the FP64 additions are left out then
// (36 or 18 instructions of 64 cycles each).  SPLIT: only the entries within
// (u, v, rz) and (w, rx, ry) count.
template <bool SPLIT>
__device__ __forceinline__ bool stage_clear(double *st, int na, int nb) {
    unsigned long long any = 0;
#pragma unroll
    for (int m = 0; m < 6; m++)
#pragma unroll
        for (int n = 0; n < 6; n += 2) {
            const bool mid = m >= 2 && m <= 4;  // rows w, rx, ry
            const bool x = !SPLIT || (mid ? n >= 2 : n == 0), y = !SPLIT || (mid ? n == 2 : n != 2);
            if (!x && !y) continue;
            const double2 o = *staged(st, na, nb, m, n);
            if (x) any |= dbits(o.x) << 1;
            if (y) any |= dbits(o.y) << 1;
        }
    return __all_sync(__activemask(), any == 0);
}

// Adds the 6x6 block K_ab of a flat isotropic element in the global frame
// (B = 0, E45 = 0, E44 = E55) onto the staged values: the non-zero terms for
// A11 = A22, A16 = A26 = 0 (same for D).  The block couples (u, v, rz) and
// (w, rx, ry) only, and each group is added as soon as it is formed.
template <bool CLEAR>
__device__ __forceinline__ void pair_add_iso(const KElem &s, const double H[3][3], const CentreH<true> &h0,
                                             double *st, int na, int nb) {
    const double A11 = s.A[0], A12 = s.A[1], ap = s.ap, am = s.am;
    // membrane and drilling: rows and columns u, v, rz
    add2<CLEAR>(st, na, nb, 0, 0, A11 * H[1][1] + ap * H[2][2], A12 * H[1][2] + am * H[2][1]);
    add2<CLEAR, false, true>(st, na, nb, 0, 4, 0., H[2][0]);
    add2<CLEAR>(st, na, nb, 1, 0, am * H[1][2] + A12 * H[2][1], ap * H[1][1] + A11 * H[2][2]);
    add2<CLEAR, false, true>(st, na, nb, 1, 4, 0., -H[1][0]);
    add2<CLEAR>(st, na, nb, 5, 0, H[0][2], -H[0][1]);
    add2<CLEAR, false, true>(st, na, nb, 5, 4, 0., H[0][0]);
    // bending and transverse shear: rows and columns w, rx, ry
    const double D11 = s.D[0], D12 = s.D[1], D66 = s.D[5], E = s.es[0];
    const double c00 = h0(0, 0);
    // The shear terms dominate and cancel in bending: each is a product rounded
    // once into its entry.  H0^xx + H0^yy summed in float-float and E c00 rounded
    // by itself save three instructions, and plate solutions lose 0.15 digits.
    const bool thick = s.flags & KF_THICK;
    const double sx = thick ? H[1][1] : h0(1, 1), sy = thick ? H[2][2] : h0(2, 2);
    add2<CLEAR>(st, na, nb, 2, 2, E * sy + E * sx, -E * h0(2, 0));
    add2<CLEAR, true, false>(st, na, nb, 2, 4, E * h0(1, 0), 0.);
    add2<CLEAR>(st, na, nb, 3, 2, -E * h0(0, 2), D66 * H[1][1] + D11 * H[2][2] + E * c00);
    add2<CLEAR, true, false>(st, na, nb, 3, 4, -(D66 * H[1][2] + D12 * H[2][1]), 0.);
    add2<CLEAR>(st, na, nb, 4, 2, E * h0(0, 1), -(D12 * H[1][2] + D66 * H[2][1]));
    add2<CLEAR, true, false>(st, na, nb, 4, 4, D11 * H[1][1] + D66 * H[2][2] + E * c00, 0.);
}

// Adds the general 6x6 block K_ab onto the staged values, three rows at a
// time.  Strains: u -> (xx, xy), v -> (xy, yy), rx -> -(xy, yy), ry -> (xx, xy)
// for the x and y derivatives (quad4.pyx:958-1000), drilling with unit weight
// d = u N_y / 2 - v N_x / 2 + rz N, shear (gyz, gxz) = (w_y - rx N, w_x + ry N).
// Of the block's 36 entries 10 are exact zeros, 18 with B = 0 (B0); elements
// evaluated in the element frame turn the 3x3 parts without multiplying them
// (FP64 instructions per lane, B = 0: 260 instead of 400), the others leave
// them out.
template <bool FF, bool B0, bool CLEAR>
__device__ __forceinline__ void pair_add_general(const KElem &s, const double H[3][3], const CentreH<FF> &h0,
                                                 double *st, int na, int nb) {
    const bool thick = s.flags & KF_THICK;
    const double E44 = s.es[0], E45 = s.es[1], E55 = s.es[2];
    const double *R = s.R, *A = s.A, *B = s.B, *D = s.D;
#pragma unroll
    for (int hb = 0; hb < 2; hb++) {
        // the rows' 3x3 parts: columns u v w and rx ry rz
        double P[3][3], Q[3][3];
        if (hb == 0) {
            const double s22 = thick ? H[2][2] : h0(2, 2), s11 = thick ? H[1][1] : h0(1, 1);
            const double s21 = thick ? H[2][1] : h0(2, 1), s12 = thick ? H[1][2] : h0(1, 2);
            P[0][0] = couple<0, 2, 0, 2>(A, s.ap, H);
            P[0][1] = couple<0, 2, 2, 1>(A, s.am, H);
            P[1][0] = couple<2, 1, 0, 2>(A, s.am, H);
            P[1][1] = couple<2, 1, 2, 1>(A, s.ap, H);
            P[2][2] = E44 * s22 + E45 * (s21 + s12) + E55 * s11;
            if (!B0) {
                Q[0][0] = -couple<0, 2, 2, 1>(B, B[5], H);
                Q[0][1] = couple<0, 2, 0, 2>(B, B[5], H);
                Q[1][0] = -couple<2, 1, 2, 1>(B, B[5], H);
                Q[1][1] = couple<2, 1, 0, 2>(B, B[5], H);
            }
            Q[0][2] = H[2][0];
            Q[1][2] = -H[1][0];
            const double h20 = h0(2, 0), h10 = h0(1, 0);
            Q[2][0] = -(E44 * h20 + E45 * h10);
            Q[2][1] = E45 * h20 + E55 * h10;
        } else {
            if (!B0) {
                P[0][0] = -couple<2, 1, 0, 2>(B, B[5], H);
                P[0][1] = -couple<2, 1, 2, 1>(B, B[5], H);
                P[1][0] = couple<0, 2, 0, 2>(B, B[5], H);
                P[1][1] = couple<0, 2, 2, 1>(B, B[5], H);
            }
            const double h02 = h0(0, 2), h01 = h0(0, 1), h00 = h0(0, 0);
            P[0][2] = -(E44 * h02 + E45 * h01);
            P[1][2] = E45 * h02 + E55 * h01;
            P[2][0] = H[0][2];
            P[2][1] = -H[0][1];
            const double e45 = E45 * h00;
            Q[0][0] = couple<2, 1, 2, 1>(D, D[5], H) + E44 * h00;
            Q[0][1] = -(couple<2, 1, 0, 2>(D, D[5], H) + e45);
            Q[1][0] = -(couple<0, 2, 2, 1>(D, D[5], H) + e45);
            Q[1][1] = couple<0, 2, 0, 2>(D, D[5], H) + E55 * h00;
            Q[2][2] = H[0][0];
        }
        if (FF) {
            if (hb == 0) {
                add2<CLEAR>(st, na, nb, 0, 0, P[0][0], P[0][1]);
                add2<CLEAR>(st, na, nb, 1, 0, P[1][0], P[1][1]);
                if (B0) {
                    add2<CLEAR, false, true>(st, na, nb, 0, 4, 0., Q[0][2]);
                    add2<CLEAR, false, true>(st, na, nb, 1, 4, 0., Q[1][2]);
                } else {
                    add2<CLEAR, false, true>(st, na, nb, 0, 2, 0., Q[0][0]);
                    add2<CLEAR, false, true>(st, na, nb, 1, 2, 0., Q[1][0]);
                    add2<CLEAR>(st, na, nb, 0, 4, Q[0][1], Q[0][2]);
                    add2<CLEAR>(st, na, nb, 1, 4, Q[1][1], Q[1][2]);
                }
                add2<CLEAR>(st, na, nb, 2, 2, P[2][2], Q[2][0]);
                add2<CLEAR, true, false>(st, na, nb, 2, 4, Q[2][1], 0.);
            } else {
                if (!B0) {
                    add2<CLEAR>(st, na, nb, 3, 0, P[0][0], P[0][1]);
                    add2<CLEAR>(st, na, nb, 4, 0, P[1][0], P[1][1]);
                }
                add2<CLEAR>(st, na, nb, 3, 2, P[0][2], Q[0][0]);
                add2<CLEAR>(st, na, nb, 4, 2, P[1][2], Q[1][0]);
                add2<CLEAR, true, false>(st, na, nb, 3, 4, Q[0][1], 0.);
                add2<CLEAR, true, false>(st, na, nb, 4, 4, Q[1][1], 0.);
                add2<CLEAR>(st, na, nb, 5, 0, P[2][0], P[2][1]);
                add2<CLEAR, false, true>(st, na, nb, 5, 4, 0., Q[2][2]);
            }
        } else {
            double tp[3][3], tq[3][3], op[3][3], oq[3][3];
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const double x = R[3 * i], y = R[3 * i + 1], z = R[3 * i + 2];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const double inP = hb == 0 || !B0 ? x * P[0][j] + y * P[1][j] : 0.;
                    const double inQ = hb == 1 || !B0 ? x * Q[0][j] + y * Q[1][j] : 0.;
                    tp[i][j] = hb == 0 ? inP : B0 ? z * P[2][j] : inP + z * P[2][j];
                    tq[i][j] = hb == 1 ? inQ : B0 ? z * Q[2][j] : inQ + z * Q[2][j];
                }
                tp[i][2] = hb == 0 ? z * P[2][2] : x * P[0][2] + y * P[1][2];
                tq[i][2] = hb == 1 ? z * Q[2][2] : x * Q[0][2] + y * Q[1][2];
            }
            turn(R, tp, op);
            turn(R, tq, oq);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                add2<CLEAR>(st, na, nb, 3 * hb + i, 0, op[i][0], op[i][1]);
                add2<CLEAR>(st, na, nb, 3 * hb + i, 2, op[i][2], oq[i][0]);
                add2<CLEAR>(st, na, nb, 3 * hb + i, 4, oq[i][1], oq[i][2]);
            }
        }
    }
}

// Phase B work of one lane: the node-pair tensor (before the caller's
// values are known to be staged) and the block added onto them (after).
__device__ __forceinline__ void pair_tensor(const KSmem &S, const KElem &s, int el, int na, int nb, double H[3][3]) {
    if (!(s.flags & KF_VALID)) return;
    if (s.flags & KF_FP64) pair_h<false>(S, el, na, nb, H);
    else pair_h<true>(S, el, na, nb, H);
}

// clear: the staged entries that the block adds to are zeros (every lane's).
__device__ __forceinline__ void pair_add(const KSmem &S, const KElem &s, int el, int na, int nb,
                                         const double H[3][3], double *st, bool clear) {
    if (!(s.flags & KF_VALID)) return;
    if (s.flags & KF_FP64) {
        const CentreH<false> h0(S, el, na, nb);
        if (s.flags & KF_B0) {
            if (clear) pair_add_general<false, true, true>(s, H, h0, st, na, nb);
            else pair_add_general<false, true, false>(s, H, h0, st, na, nb);
        } else {
            if (clear) pair_add_general<false, false, true>(s, H, h0, st, na, nb);
            else pair_add_general<false, false, false>(s, H, h0, st, na, nb);
        }
    } else {
        const CentreH<true> h0(S, el, na, nb);
        if (s.flags & KF_ISO) {
            if (clear) pair_add_iso<true>(s, H, h0, st, na, nb);
            else pair_add_iso<false>(s, H, h0, st, na, nb);
        } else if (s.flags & KF_B0) {
            if (clear) pair_add_general<true, true, true>(s, H, h0, st, na, nb);
            else pair_add_general<true, true, false>(s, H, h0, st, na, nb);
        } else {
            if (clear) pair_add_general<true, false, true>(s, H, h0, st, na, nb);
            else pair_add_general<true, false, false>(s, H, h0, st, na, nb);
        }
    }
}

// Phase B of one round for a warp: the tile's elements el0 (lanes 0-15) and
// el0 + 1 (lanes 16-31), one lane per node pair: the caller's current values
// are prefetched into stage[0..1] with cp.async while the 6x6 blocks are
// computed, then the blocks are added onto them (ready for the write-out).
__device__ __forceinline__ void kc0_round(const Q4Args &a, KSmem &S, const KElem *els, int el0,
                                          double (*stage)[24 * KROW], int lane) {
    const int half = lane >> 4, pair = lane & 15;
    const int na = pair >> 2, nb = pair & 3;
    const int el = el0 + half;
    double *st = stage[half];
    // prefetch the two elements' current values into the stage
#pragma unroll
    for (int hh = 0; hh < 2; hh++) {
        const KElem &t = els[el0 + hh];
        if (!(t.flags & KF_VALID)) continue;
        const double *kv = a.Kv + t.init_k;
        double *sv = stage[hh];
        if (a.vec16 && !(t.init_k & 1)) {
            // 16-byte pieces: slots 2 lane + 64 j, j = 0..8
            int row = lane / 12, col = 2 * lane - 24 * row;
#pragma unroll 3
            for (int j = 0; j < 9; j++) {
                cp_async16(sv + row * KROW + col, kv + 2 * lane + 64 * j);
                col += 16;
                row += 2;
                if (col >= 24) {
                    col -= 24;
                    row += 1;
                }
            }
        } else {
#pragma unroll 6
            for (int i = lane; i < 576; i += 32) {
                const int row = i / 24, col = i - row * 24;
                cp_async8(sv + row * KROW + col, kv + i);
            }
        }
    }
    cp_async_commit();
    double H[3][3];
    pair_tensor(S, els[el], el, na, nb, H);
    // all lanes' prefetches of both staged elements have landed
    cp_async_wait_all();
    __syncwarp();
    const KElem &s = els[el];
    const bool clear = (s.flags & KF_SPLIT) ? stage_clear<true>(st, na, nb) : stage_clear<false>(st, na, nb);
    pair_add(S, s, el, na, nb, H, st, clear);
    __syncwarp();
}

// Phase A2 for element slot el at point g: w detJ and the shape functions
// with their Cartesian derivatives (float-float for flat elements, FP64
// otherwise).
__device__ __forceinline__ void kc0_point(KSmem &S, const KElem &s, int el, int g) {
    if (!(s.flags & KF_VALID)) return;
    Slot *o = S.gp[el][g];
    if (s.flags & KF_FP64) {
        double xi, eta, detJ, N[4], Nx[4], Ny[4], xy[8];
#pragma unroll
        for (int i = 0; i < 8; i++) xy[i] = s.xy[i].d;
        point_coords(g, xi, eta);
        quad_derivs(xy, xi, eta, detJ, N, Nx, Ny);
        o[0].d = (g == 4) ? 4. * detJ : detJ;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            o[1 + i].d = Nx[i];
            o[5 + i].d = Ny[i];
        }
    } else {
        point_ff(s, S.shape, g, o);
    }
}

// The per-CTA copy of the float-float shape-function table.
__device__ __forceinline__ void kc0_tables(KSmem &S, int tid) {
    for (int i = tid; i < KPTS * 12; i += KNT) (&S.shape[0][0][0])[i] = (&c_shape[0][0][0])[i];
}

// Phase A2 of a consumer warp: the points of its per (2 or 4) elements from
// el0 on, one lane each.
__device__ __forceinline__ void kc0_points(KSmem &S, const KElem *els, int el0, int per, int lane) {
    if (lane < per * KPTS) kc0_point(S, els[el0 + lane / KPTS], el0 + lane / KPTS, lane % KPTS);
    __syncwarp();
}

// The tiles of a CTA over cnt elements: full tiles of KT, interleaved over the
// CTAs, then one smaller tile each that shares what is left evenly.
struct KTiles {
    int64_t full, rest0, left;
    __device__ __forceinline__ KTiles(int64_t cnt) {
        full = cnt / ((int64_t)KT * gridDim.x);
        rest0 = full * KT * gridDim.x;
        left = cnt - rest0;
    }
    // first element and number of elements of the CTA's t-th tile (0: none)
    __device__ __forceinline__ int64_t first(int64_t t) const {
        return t < full ? (t * gridDim.x + blockIdx.x) * KT : rest0 + left * blockIdx.x / gridDim.x;
    }
    __device__ __forceinline__ int count(int64_t t) const {
        if (t < full) return KT;
        return t > full ? 0 : (int)(left * (blockIdx.x + 1) / gridDim.x - left * blockIdx.x / gridDim.x);
    }
};

__global__ void __launch_bounds__(KNT, KMINB) quad4_kc0_ff_kernel(Q4Args a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    KSmem &S = *reinterpret_cast<KSmem *>(smem_raw);
    const int tid = threadIdx.x;
    kc0_tables(S, tid);
    const int lane = tid & 31, warp = tid >> 5;
    const KTiles tiles(a.E);
    // the last warp runs phase A one tile ahead of the others
    auto phase_a = [&](int64_t t, int buf) {
        if (warp != KCW || lane >= KT) return;
        if (lane < tiles.count(t)) kc0_phase_a2(a, tiles.first(t) + lane, S.el[buf][lane]);
        else S.el[buf][lane].flags = 0;
    };
    phase_a(0, 0);
    int buf = 0, n;
    for (int64_t t = 0; (n = tiles.count(t)) > 0; t++, buf ^= 1) {
        __syncthreads();
        if (warp == KCW) {
            phase_a(t + 1, buf ^ 1);
            continue;
        }
        const int per = n > 2 * KCW ? 4 : 2, first = warp * per;
        if (first >= n) continue;
        const KElem *els = S.el[buf];
        kc0_points(S, els, first, per, lane);
        for (int el0 = first; el0 < first + per && el0 < n; el0 += 2) {
            kc0_round(a, S, els, el0, S.stage[warp], lane);
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                const KElem &e = els[el0 + hh];
                if (e.flags & KF_VALID) write_staged(a, S.stage[warp][hh], e.init_k, e.c, lane);
            }
            __syncwarp();
        }
    }
}


// ------------------------------------------------------ CSR write-out mode
// The same element computation with the blocks sent straight to the reduced
// CSR values through an element -> CSR scatter map (fused.cu): one launch
// per element colour (no two elements of a colour share a node), so the
// read-add-write of the CSR entries needs no atomics and sums every entry
// in a fixed order.  The node-pair blocks an element assigns (it is their
// first contributor) are stored without reading, and where a warp's blocks are
// all assigned nothing is added.
//
// Bound by latency and instructions (1,261 per element on interior isotropic
// elements, 2,123 with a test, a position and a bounds check per row and
// entry), then by the colours' passes over the values (3 TB/s).  90,000
// elements in 4 colours 0.50 -> 0.33 ms.

struct CsrArgs {
    const int32_t *order;  // the colour's elements
    int64_t cnt;
    const int32_t *node;   // [E, 4] node indices
    const int32_t *boff;   // [E, 16] offsets of node j's columns in node i's rows
    const uint32_t *first; // [E] assign bits
    const fe3d_noderow *nr;
    int64_t nnodes;
    double *vals;
    int64_t nnz;
    int assign;
    int atomic;  // one launch over all elements, blocks added with atomics (order unspecified)
};

// Per element of the tile: row length | free mask << 16 of its nodes, the
// block offsets and the assign bits (the nodes' row starts go to KElem.c).
struct __align__(8) CsrElem {
    int Lf[4];
    short boff[16];
    unsigned first;
    int pad;
};

struct KSmemCsr {
    KSmem s;
    CsrElem cm[2][KT];
};

// KMINB CTAs per SM must fit the SM's 228 KB of shared memory (1 KB of it
// reserved per CTA)
static_assert(KMINB * (sizeof(KSmem) + 1024) <= 228 * 1024, "triplet kernel: shared memory per SM");
static_assert(KMINB * (sizeof(KSmemCsr) + 1024) <= 228 * 1024, "CSR kernel: shared memory per SM");

__device__ void kc0_phase_a_csr(const Q4Args &a, const CsrArgs &m, int64_t t, KElem &s, CsrElem &q) {
    s.flags = 0;
    const int64_t e = m.order ? (int64_t)m.order[t] : t;
    int32_t nd[4];
    bool ok = e >= 0 && e < a.E;
    if (ok) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            nd[i] = m.node[4 * e + i];
            ok &= nd[i] >= 0 && nd[i] < m.nnodes;
        }
    }
    if (!ok) {
        raise_error(a.err, kErrBounds);
        return;
    }
    long long c[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        c[i] = 6LL * nd[i];
        const fe3d_noderow r = m.nr[nd[i]];
        s.c[i] = r.rs;
        q.Lf[i] = r.L | (r.fm << 16);
    }
    const int4 *bo = reinterpret_cast<const int4 *>(m.boff + 16 * e);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int4 v = bo[k];
        q.boff[4 * k] = (short)v.x;
        q.boff[4 * k + 1] = (short)v.y;
        q.boff[4 * k + 2] = (short)v.z;
        q.boff[4 * k + 3] = (short)v.w;
    }
    q.first = m.assign ? m.first[e] : 0u;
    s.init_k = 0;
    // every row and column of the element inside the values
    bool all = true;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int fm = q.Lf[i] >> 16, L = q.Lf[i] & 0xffff;
        all &= fm == 63;
        if (fm) ok &= s.c[i] >= 0 && s.c[i] + (long long)__popc(fm) * L <= m.nnz;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (fm) ok &= q.boff[4 * i + j] >= 0 && q.boff[4 * i + j] + __popc(q.Lf[j] >> 16) <= L;
    }
    kc0_elem_setup(a, e, c, ok, s);
    if (all && (s.flags & KF_VALID)) s.flags |= KF_FREE;
}

// The entries of a staged element that move: lane l < 24 takes column l (column
// n of node b) for the free rows of the four nodes, f(stage index, address)
// each, in warp-wide accesses of a node's runs of columns.  The rows of a node
// are L entries apart, so a lane forms one address per node.  Elements that do
// not couple (u, v, rz) and (w, rx, ry) move a lane's three rows of its own
// group; the other three are exact zeros, which only assigned blocks store:
// z(address).  skip(assigned) leaves a node's rows out.
template <class S, class F, class Z>
__device__ __forceinline__ void csr_entries(const CsrArgs &m, const KElem &t, const CsrElem &q, int lane, S &&skip,
                                            F &&f, Z &&z) {
    const int b = lane / 6, n = lane - 6 * b;
    if (lane >= 24 || !(t.flags & KF_VALID)) return;
    const bool mid = n >= 2 && n <= 4;
    if ((t.flags & (KF_SPLIT | KF_FREE)) == (KF_SPLIT | KF_FREE)) {
        // the three rows of the lane's group and of the other one
        const int i0 = mid ? 2 : 0, i2 = mid ? 4 : 5, o0 = mid ? 0 : 2, o2 = mid ? 5 : 4;
#pragma unroll
        for (int a = 0; a < 4; a++) {
            const bool asg = (q.first >> (4 * a + b)) & 1;
            if (skip(asg)) continue;
            const int L = q.Lf[a] & 0xffff, si = 6 * a * KROW + lane;
            double *p = m.vals + (t.c[a] + q.boff[4 * a + b] + n);
            double *p0 = p + i0 * L;
            f(si + i0 * KROW, p0);
            f(si + (i0 + 1) * KROW, p0 + L);
            f(si + i2 * KROW, p + i2 * L);
            if (asg) {
                double *z0 = p + o0 * L;
                z(z0);
                z(z0 + L);
                z(p + o2 * L);
            }
        }
        return;
    }
    const int fb = q.Lf[b] >> 16;
    if (!((fb >> n) & 1)) return;  // fixed column
    const int rank = __popc(fb & ((1 << n) - 1));
    const bool split = t.flags & KF_SPLIT;
#pragma unroll 1
    for (int a = 0; a < 4; a++) {
        const bool asg = (q.first >> (4 * a + b)) & 1;
        const int Lf = q.Lf[a], fm = Lf >> 16, L = Lf & 0xffff;
        if (skip(asg) || !fm) continue;
        double *p = m.vals + (t.c[a] + q.boff[4 * a + b] + rank);
#pragma unroll
        for (int i = 0; i < 6; i++) {
            if (!((fm >> i) & 1)) continue;
            if (split && (i >= 2 && i <= 4) != mid) {
                if (asg) z(p);
            } else {
                f((6 * a + i) * KROW + lane, p);
            }
            p += L;
        }
    }
}

// Current values of the blocks that are added to.
__device__ __forceinline__ void csr_prefetch(const CsrArgs &m, const KElem &t, const CsrElem &q, double *sv,
                                             int lane) {
    if (m.atomic) return;
    csr_entries(m, t, q, lane, [](bool asg) { return asg; }, [&](int si, double *p) { cp_async8(sv + si, p); },
                [](double *) {});
}

// Stores the staged entries (assigned blocks with their exact zeros, which the
// stage does not hold), or adds them with atomics.
__device__ __forceinline__ void csr_write(const CsrArgs &m, const KElem &t, const CsrElem &q, const double *sv,
                                          int lane) {
    if (m.atomic)
        csr_entries(m, t, q, lane, [](bool) { return false; },
                    [&](int si, double *p) { atomicAdd(p, sv[si]); }, [](double *) {});
    else
        csr_entries(m, t, q, lane, [](bool) { return false; }, [&](int si, double *p) { *p = sv[si]; },
                    [](double *p) { *p = 0.; });
}

__device__ __forceinline__ void kc0_round_csr(const Q4Args &a, const CsrArgs &m, KSmem &S, const KElem *els,
                                              const CsrElem *cm, int el0, double (*stage)[24 * KROW], int lane) {
    const int half = lane >> 4, pair = lane & 15;
    const int na = pair >> 2, nb = pair & 3;
    const int el = el0 + half;
    const KElem &s = els[el];
    double *st = stage[half];
#pragma unroll
    for (int hh = 0; hh < 2; hh++) csr_prefetch(m, els[el0 + hh], cm[el0 + hh], stage[hh], lane);
    cp_async_commit();
    double H[3][3];
    pair_tensor(S, s, el, na, nb, H);
    cp_async_wait_all();
    __syncwarp();
    // a block that is assigned (or added with atomics) starts from zeros; a
    // warp with such blocks only makes no additions
    const bool own = m.atomic || ((cm[el].first >> (4 * na + nb)) & 1);
    const bool clear = __all_sync(0xffffffffu, own || !(s.flags & KF_VALID));
    if (own && !(clear && (s.flags & (KF_SPLIT | KF_FP64))))
#pragma unroll
        for (int i = 0; i < 6; i++)
#pragma unroll
            for (int j = 0; j < 6; j += 2) *staged(st, na, nb, i, j) = make_double2(0., 0.);
    pair_add(S, s, el, na, nb, H, st, clear);
    __syncwarp();
}

__global__ void __launch_bounds__(KNT, KMINB) quad4_kc0_csr_kernel(Q4Args a, CsrArgs m) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    KSmemCsr &SC = *reinterpret_cast<KSmemCsr *>(smem_raw);
    KSmem &S = SC.s;
    const int tid = threadIdx.x;
    kc0_tables(S, tid);
    const int lane = tid & 31, warp = tid >> 5;
    const KTiles tiles(m.cnt);
    auto phase_a = [&](int64_t t, int buf) {
        if (warp != KCW || lane >= KT) return;
        if (lane < tiles.count(t)) kc0_phase_a_csr(a, m, tiles.first(t) + lane, S.el[buf][lane], SC.cm[buf][lane]);
        else S.el[buf][lane].flags = 0;
    };
    phase_a(0, 0);
    // the next colour's CTAs may start as these end; this colour's values wait
    // for the previous one (both no-ops in a launch without the attribute)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int buf = 0, n;
    for (int64_t t = 0; (n = tiles.count(t)) > 0; t++, buf ^= 1) {
        __syncthreads();
        if (warp == KCW) {
            phase_a(t + 1, buf ^ 1);
            continue;
        }
        const int per = n > 2 * KCW ? 4 : 2, first = warp * per;
        if (first >= n) continue;
        const KElem *els = S.el[buf];
        kc0_points(S, els, first, per, lane);
        for (int el0 = first; el0 < first + per && el0 < n; el0 += 2) {
            kc0_round_csr(a, m, S, els, SC.cm[buf], el0, S.stage[warp], lane);
#pragma unroll
            for (int hh = 0; hh < 2; hh++)
                csr_write(m, els[el0 + hh], SC.cm[buf][el0 + hh], S.stage[warp][hh], lane);
            __syncwarp();
        }
    }
}

// One wave of CTAs; small meshes spread over the SMs (4 elements a CTA).
int kc0_grid(int64_t E) {
    const int64_t g = (E + 3) / 4, cap = (int64_t)kSMs * KMINB;
    return (int)(g < cap ? g : cap);
}

int g_shape_ready[64] = {0};

int upload_shape_table() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return FE3D_ERR_CUDA;
    if (dev < 64 && g_shape_ready[dev]) return FE3D_OK;
    ff h[KPTS][3][4];
    const double sx[4] = {-1., 1., 1., -1.}, sy[4] = {-1., -1., 1., 1.};
    for (int g = 0; g < KPTS; g++) {
        double xi, eta;
        if (g == 4) {
            xi = 0.;
            eta = 0.;
        } else {
            xi = (g & 2) ? kGauss : -kGauss;
            eta = (g & 1) ? kGauss : -kGauss;
        }
        for (int i = 0; i < 4; i++) {
            const double v[3] = {0.25 * (1 + sx[i] * xi) * (1 + sy[i] * eta), 0.25 * sx[i] * (1 + sy[i] * eta),
                                 0.25 * sy[i] * (1 + sx[i] * xi)};
            for (int t = 0; t < 3; t++) {
                const float hi = (float)v[t];
                h[g][t][i] = {hi, (float)(v[t] - (double)hi)};
            }
        }
    }
    if (cudaMemcpyToSymbol(c_shape, h, sizeof(h)) != cudaSuccess) return FE3D_ERR_CUDA;
    if (cudaFuncSetAttribute(quad4_kc0_ff_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(KSmem)) != cudaSuccess ||
        cudaFuncSetAttribute(quad4_kc0_csr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(KSmemCsr)) != cudaSuccess)
        return FE3D_ERR_CUDA;
    if (dev < 64) g_shape_ready[dev] = 1;
    return FE3D_OK;
}

}  // namespace
}  // namespace fe3d

using namespace fe3d;

extern "C" int fe3d_quad4_kc0(int64_t E, const int64_t *cdof, const int64_t *init_k,
                              const double *x, int64_t nx, const double *xmat, int xmat_stride,
                              const double *R, const double *m, const double *xe,
                              const double *area, const double *props, int64_t nprops,
                              const int32_t *pid, int64_t *Kr, int64_t *Kc, double *Kv, int64_t nk,
                              int values_only, int *err, void *stream) {
    if (E < 0) return FE3D_ERR_ARG;
    if (E == 0) return FE3D_OK;
    if (!cdof || !init_k || !props || !Kv || nprops <= 0) return FE3D_ERR_ARG;
    if (!values_only && (!Kr || !Kc)) return FE3D_ERR_ARG;
    if (!x && (!R || !m || !xe || !area)) return FE3D_ERR_ARG;
    if (xmat && xmat_stride != 0 && xmat_stride != 3) return FE3D_ERR_ARG;
    const int rc = upload_shape_table();
    if (rc) return rc;
    Q4Args a{E, cdof, init_k, x, nx, xmat, xmat_stride, R, m, xe, area, props, nprops, pid,
             Kr, Kc, Kv, nk, values_only, err};
    // 16-byte write-out for elements with an even init_k when the output
    // arrays are 16-byte aligned
    const auto al16 = [](const void *q) { return ((uintptr_t)q & 15u) == 0; };
    a.vec16 = al16(Kv) && (values_only || (al16(Kr) && al16(Kc)));
    quad4_kc0_ff_kernel<<<kc0_grid(E), KNT, sizeof(KSmem), as_stream(stream)>>>(a);
    FE3D_CHECK_LAUNCH();
    return FE3D_OK;
}

extern "C" int fe3d_quad4_kc0_csr(const fe3d_fmap *fm, int g, const double *x, int64_t nx, const double *xmat,
                                  int xmat_stride, const double *props, int64_t nprops, const int32_t *pid,
                                  double *vals, int mode, int *err, void *stream) {
    if (!fm || g < 0 || g >= fm->ngroups ||
        (mode != FE3D_CSR_ADD && mode != FE3D_CSR_ASSIGN && mode != FE3D_CSR_ATOMIC))
        return FE3D_ERR_ARG;
    const fe3d_fmap_group &G = fm->g[g];
    if (G.nn != 4) return FE3D_ERR_ARG;
    if (G.E == 0 || fm->pat->nnz == 0) return FE3D_OK;
    if (!x || !props || nprops <= 0 || !vals) return FE3D_ERR_ARG;
    if (xmat && xmat_stride != 0 && xmat_stride != 3) return FE3D_ERR_ARG;
    if (fm->pat->max_row_len > 32767) return FE3D_ERR_ARG;  // block offsets are staged as int16
    const int rc = upload_shape_table();
    if (rc) return rc;
    Q4Args a{G.E, nullptr, nullptr, x, nx, xmat, xmat_stride, nullptr, nullptr, nullptr, nullptr, props, nprops, pid,
             nullptr, nullptr, nullptr, 0, 1, err};
    a.vec16 = 0;
    if (mode == FE3D_CSR_ATOMIC) {
        CsrArgs m{nullptr, G.E, G.node, G.boff, G.first, fm->pat->noderow, fm->pat->nnodes,
                  vals, fm->pat->nnz, 0, 1};
        quad4_kc0_csr_kernel<<<kc0_grid(G.E), KNT, sizeof(KSmemCsr), as_stream(stream)>>>(a, m);
        FE3D_CHECK_LAUNCH();
        return FE3D_OK;
    }
    bool launched = false;
    for (int c = 0; c < G.ncolors; c++) {
        const int64_t cnt = G.cstart[c + 1] - G.cstart[c];
        if (cnt == 0) continue;
        CsrArgs m{G.order + G.cstart[c], cnt, G.node, G.boff, G.first, fm->pat->noderow, fm->pat->nnodes,
                  vals, fm->pat->nnz, mode == FE3D_CSR_ASSIGN, 0};
        // colours after the first overlap their set-up with the tail of the one
        // before; the first waits for whatever the caller has queued
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kc0_grid(cnt));
        cfg.blockDim = dim3(KNT);
        cfg.dynamicSmemBytes = sizeof(KSmemCsr);
        cfg.stream = as_stream(stream);
        cfg.attrs = &at;
        cfg.numAttrs = launched ? 1 : 0;
        if (cudaLaunchKernelEx(&cfg, quad4_kc0_csr_kernel, a, m) != cudaSuccess) return FE3D_ERR_LAUNCH;
        launched = true;
    }
    return FE3D_OK;
}
