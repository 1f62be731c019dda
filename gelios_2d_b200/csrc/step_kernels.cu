// sm_100a kernels of the Gelios_2D plasma time step.
//
// One time step of Setka::Go_5_komponent__MK2 (Setka.cpp:10121-10482) is,
// on several streams:
//   mk2_recon_tracked_kernel  TVD states of the tracked face units (pre-motion)
//   mk2_tracked_solve_kernel  star pressures of the tracked faces' exact
//                             Riemann problems (warp per face)
//   mk2_source_kernel         charge-exchange source (Get_Sourse_MK1), 32
//                             cells per warp: a cell phase (one lane per
//                             cell), then a species phase (one lane per cell
//                             and hydrogen species)
//   surface_faces_kernel      Move_surface (Setka.cpp:3378-3844): exact
//                             Godunov speeds of the tracked faces (warp per
//                             face)
//   rails_kernel              node velocities of the key points, then
//                             Move_Setka_Calculate_2 (Setka.cpp:4324-4759):
//                             one CTA per rail
//   mk2_flux_tracked_kernel   tracked faces: HLL + the Riemann solution
//                             sampled at the moved face speed
//   mk2_face_kernel           reconstruction and HLL flux of the plain interior
//                             face units (face speed from the moved points),
//                             F.S once per unit; CFL block-min
//   mk2_face_rest_kernel      the C_1 interior and the one-sided units
//   mk2_update_kernel         a cell's fluxes summed in Grans order, the
//                             conservative ALE update, the next step's
//                             geometry cache
//   commit_kernel             x = x2; dt of the next step (the last step of a
//                             call; within one the surface kernel finalises dt)
// (mk2_tile_kernel, one tile of cells per block with the fluxes in shared
// memory, is the other arrangement of the last four.)
// Go_stationary (Setka.cpp:5205-5343) is stationary_lanes_kernel (four lanes
// per cell, every step of a call) or, where that does not take the grid,
// stationary_persistent_kernel; Go_stationary_5_komponent_inner_MK2
// (Setka.cpp:6999-7212) is inner_table_kernel + inner_lanes_kernel, or
// inner_cell_kernel + dt_finalize_kernel.
//
// A cell's faces are summed by one thread or one group of lanes in the
// reference's Grans order, so no floating-point atomics are needed and results
// are deterministic run to run.  The CFL minimum is exact under any order
// (atomicMin on the bit pattern of non-negative doubles).
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include <cooperative_groups.h>

#include "physics.cuh"
#include "plain_plan.cuh"
#include "step_kernels.cuh"

namespace cg = cooperative_groups;

// Minimum resident blocks per SM of the grid-wide moving-grid kernels
// (register caps: 128 threads x 65536/(128 x minBlocks) registers).
#ifndef GELIOS_SOURCE_MINB
#define GELIOS_SOURCE_MINB 10
#endif

namespace gelios {

// ------------------------------------------------------------------ helpers
__device__ __forceinline__ St5 load_state(const double* const* st, int c) {
    St5 s;
    s.ro = st[0][c];
    s.p = st[1][c];
    s.u = st[2][c];
    s.v = st[3][c];
    s.Q = st[4][c];
    return s;
}

// Cell::Get_Center (Cell.cpp:66-88) on coordinates X, Y.
__device__ __forceinline__ void centroid(const int32_t* contour, int n, const double* X, const double* Y, double& ox,
                                         double& oy) {
    double A = 0.0, Gx = 0.0, Gy = 0.0;
    int a = contour[0];
    double xa = X[a], ya = Y[a];
    const double x0 = xa, y0 = ya;
    for (int i = 0; i < n; i++) {
        double xb, yb;
        if (i + 1 == n) {
            xb = x0;
            yb = y0;
        } else {
            const int b = contour[i + 1];
            xb = X[b];
            yb = Y[b];
        }
        const double cr = xa * yb - ya * xb;
        A = A + cr;
        Gx = Gx + (xa + xb) * cr;
        Gy = Gy + (ya + yb) * cr;
        xa = xb;
        ya = yb;
    }
    A = A * 0.5;
    ox = Gx / (6.0 * A);
    oy = Gy / (6.0 * A);
}

// Cell::Get_Volume_rotate(360)/(2 pi) (Cell.cpp:188-206) on X, Y.
__device__ __forceinline__ double volume_rotate(const int32_t* contour, int n, const double* X, const double* Y) {
    double A = 0.0, G = 0.0;
    int a = contour[0];
    double xa = X[a], ya = Y[a];
    const double x0 = xa, y0 = ya;
    for (int i = 0; i < n; i++) {
        double xb, yb;
        if (i + 1 == n) {
            xb = x0;
            yb = y0;
        } else {
            const int b = contour[i + 1];
            xb = X[b];
            yb = Y[b];
        }
        const double cr = xa * yb - ya * xb;
        A = A + cr;
        G = G + (ya + yb) * cr;
        xa = xb;
        ya = yb;
    }
    A = A * 0.5;
    return fabs(A) * (1.0 / (6.0 * A)) * G * kPi * 360.0 / 180.0 / (2.0 * kPi);
}

// Cell::Get_Volume / Get_Volume_posle (Cell.cpp:146-186, 208-254).
// posle selects the arithmetic-mean centre of the non-quad branch.
__device__ double area(const int32_t* contour, int n, const int32_t* sA, const int32_t* sB, int g0, int g1,
                       const double* X, const double* Y, bool posle) {
    if (n == 4) {
        const int p0 = contour[0], p1 = contour[1], p2 = contour[2], p3 = contour[3];
        double a1 = X[p0] - X[p2];
        double a2 = Y[p0] - Y[p2];
        const double a = sqrt(sq(a1) + sq(a2));
        double b1 = X[p1] - X[p3];
        double b2 = Y[p1] - Y[p3];
        const double b = sqrt(sq(b1) + sq(b2));
        a1 = a1 / a;
        a2 = a2 / a;
        b1 = b1 / b;
        b2 = b2 / b;
        const double c = a1 * b1 + a2 * b2;
        const double s = sqrt(1 - sq(c));
        return 0.5 * a * b * s;
    }
    double x = 0.0, y = 0.0;
    if (!posle) {
        centroid(contour, n, X, Y, x, y);
    } else {
        for (int i = 0; i < n; i++) {
            x += X[contour[i]];
            y += Y[contour[i]];
        }
        x = x / (1.0 * n);
        y = y / (1.0 * n);
    }
    double S = 0.0;
    for (int g = g0; g < g1; g++) {
        const int pa = sA[g], pb = sB[g];
        const double a1 = sqrt(sq(X[pa] - x) + sq(Y[pa] - y));
        const double a2 = sqrt(sq(X[pb] - x) + sq(Y[pb] - y));
        const double a3 = sqrt(sq(X[pa] - X[pb]) + sq(Y[pa] - Y[pb]));
        const double p = (a1 + a2 + a3) / 2.0;
        S = S + sqrt(p * (p - a1) * (p - a2) * (p - a3));
    }
    return S;
}

// centroid, area (Get_Volume) and rotated volume of a quadrilateral whose
// corners (contour order) are in registers: the operations of centroid(),
// area() (n == 4) and volume_rotate() in the same order.
__device__ __forceinline__ void quad_geometry(const double (&X)[4], const double (&Y)[4], double& ox, double& oy,
                                              double& vs, double& vol) {
    double A = 0.0, Gx = 0.0, Gy = 0.0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const double xa = X[i], ya = Y[i], xb = X[(i + 1) & 3], yb = Y[(i + 1) & 3];
        const double cr = xa * yb - ya * xb;
        A = A + cr;
        Gx = Gx + (xa + xb) * cr;
        Gy = Gy + (ya + yb) * cr;
    }
    A = A * 0.5;
    ox = Gx / (6.0 * A);
    oy = Gy / (6.0 * A);
    vol = fabs(A) * (1.0 / (6.0 * A)) * Gy * kPi * 360.0 / 180.0 / (2.0 * kPi);
    double a1 = X[0] - X[2];
    double a2 = Y[0] - Y[2];
    const double a = sqrt(sq(a1) + sq(a2));
    double b1 = X[1] - X[3];
    double b2 = Y[1] - Y[3];
    const double bb = sqrt(sq(b1) + sq(b2));
    a1 = a1 / a;
    a2 = a2 / a;
    b1 = b1 / bb;
    b2 = b2 / bb;
    const double cc = a1 * b1 + a2 * b2;
    const double sn = sqrt(1 - sq(cc));
    vs = 0.5 * a * bb * sn;
}

// The same for the moving-grid update: the area as half the cross product of
// the diagonals (the reference's |d1| |d2| sin(angle) / 2 without its three
// square roots and four quotients; it rounds less, its sine loses digits
// where the diagonals are nearly parallel) and one reciprocal.
__device__ __forceinline__ void quad_geometry_lean(const double (&X)[4], const double (&Y)[4], double& ox, double& oy,
                                                   double& vs, double& vol) {
    double A = 0.0, Gx = 0.0, Gy = 0.0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const double xa = X[i], ya = Y[i], xb = X[(i + 1) & 3], yb = Y[(i + 1) & 3];
        const double cr = xa * yb - ya * xb;
        A = A + cr;
        Gx = Gx + (xa + xb) * cr;
        Gy = Gy + (ya + yb) * cr;
    }
    const double r = 1.0 / (3.0 * A);  // 1 / (6 area)
    ox = Gx * r;
    oy = Gy * r;
    vol = fabs(0.5 * A) * r * Gy * kPi * 360.0 / 180.0 / (2.0 * kPi);
    vs = 0.5 * fabs((X[0] - X[2]) * (Y[1] - Y[3]) - (Y[0] - Y[2]) * (X[1] - X[3]));
}

// Inner_sphere BC state (Gran.cpp:234-265, 520-534) at face centre (x, y).
__device__ __forceinline__ St5 inner_sphere_state(const gelios_params& P, double x, double y) {
    const double dist = sqrt(x * x + y * y);
    const double ro = 1.0 / (sq(P.chi) * dist * dist);
    const double P_E = ro * P.chi * P.chi / (P.gamma * P.inner_mach * P.inner_mach);
    St5 s;
    s.ro = ro;
    s.p = P_E;
    s.u = P.chi * x / dist;
    s.v = P.chi * y / dist;
    s.Q = ro;
    return s;
}
__device__ __forceinline__ St5 input_state(const gelios_params& P) {
    St5 s;
    s.ro = P.in_ro;
    s.p = P.in_p;
    s.u = P.in_u;
    s.v = P.in_v;
    s.Q = P.in_Q;
    return s;
}

// Gran::Get_par (Gran.cpp:205-289) for a face of the owning cell `own`.
__device__ __forceinline__ St5 get_par(const gelios_params& P, int ft, const St5& own, const double* const* st,
                                       int nb, double fx, double fy) {
    St5 s = own;
    if (ft == G_USUALY) {
        s = load_state(st, nb);
    } else if (ft == G_EXTERN) {
        if (s.u >= 0.0) s.u = P.extern_u_par;
    } else if (ft == G_AXIS) {
        s.v = -s.v;
    } else if (ft == G_INNER_SPHERE) {
        s = inner_sphere_state(P, fx, fy);
    } else if (ft == G_INPUT) {
        s = input_state(P);
    }
    return s;
}

// dM, dS: distances from the face centre to the centroids of M and So (the
// face unit computes them for its CFL candidates; passed in, not recomputed).
__device__ St5 tvd_usualy_d(const double* const* st, const double* cx, const double* cy, double fx, double fy,
                            const St5& Ms, double Mx, double My, int So, int Sd, bool m_has_axis, bool tracked,
                            double dM, double dS, int* status) {
    if (Sd < 0) {
        St5 par = Ms;
        if (m_has_axis) {  // Gran.cpp:308-338
            const St5 par3 = load_state(st, So);
            const double dist2 = dM;
            const double dist3 = dS;
            const double dist1 = sqrt(sq(fx - Mx) + sq(fy - (-My)));
            par.v = linear3(-dist1, -Ms.v, -dist2, Ms.v, dist3, par3.v, 0.0);
        }
        return par;
    }
    const St5 par1 = load_state(st, Sd);
    const double dist2 = dM;
    if (tracked) {  // Gran.cpp:345-426
        const double dist1 = sqrt(sq(fx - cx[Sd]) + sq(fy - cy[Sd]));
        // linear(-dist1, t1, -dist2, t2, 0) with one reciprocal
        const double r = 1.0 / (-dist1 - (-dist2)), x2 = -dist2;
        St5 o;
        o.ro = (par1.ro - Ms.ro) * r * (0.0 - x2) + Ms.ro;
        o.p = (par1.p - Ms.p) * r * (0.0 - x2) + Ms.p;
        o.u = (par1.u - Ms.u) * r * (0.0 - x2) + Ms.u;
        o.v = (par1.v - Ms.v) * r * (0.0 - x2) + Ms.v;
        o.Q = (par1.Q - Ms.Q) * r * (0.0 - x2) + Ms.Q;
        if (o.ro <= 0.0) o.ro = Ms.ro;
        if (o.p <= 0.0) o.p = Ms.p;
        return o;
    }
    const St5 par3 = load_state(st, So);
    const double dist3 = dS;
    const double dist1 = sqrt(sq(fx - cx[Sd]) + sq(fy - cy[Sd]));
    // linear(-dist1, t1, -dist2, t2, dist3, t3, 0) for the five fields
    const double r12 = 1.0 / (-dist1 - (-dist2)), r23 = 1.0 / (-dist2 - dist3), x2 = -dist2;
    St5 o;
    o.ro = linear3r(par1.ro, Ms.ro, par3.ro, r12, r23, x2);
    o.p = linear3r(par1.p, Ms.p, par3.p, r12, r23, x2);
    o.u = linear3r(par1.u, Ms.u, par3.u, r12, r23, x2);
    o.v = linear3r(par1.v, Ms.v, par3.v, r12, r23, x2);
    o.Q = linear3r(par1.Q, Ms.Q, par3.Q, r12, r23, x2);
    if (o.ro <= 0.0 || o.p <= 0.0) *status |= ST_TVD_BAD;  // the reference exits (Gran.cpp:444-455)
    return o;
}

// Gran::Get_par_TVD (Gran.cpp:292-473) of a Usualy face seen from Master M
// (state Ms, centre Mx,My) with Sosed So and Sosed_down Sd.
__device__ St5 tvd_usualy(const double* const* st, const double* cx, const double* cy, double fx, double fy,
                          const St5& Ms, double Mx, double My, int So, int Sd, bool m_has_axis, bool tracked,
                          int* status) {
    const double dM = sqrt(sq(fx - Mx) + sq(fy - My));
    const double dS = (Sd < 0 && !m_has_axis) || (Sd >= 0 && tracked) ? 0.0 : sqrt(sq(fx - cx[So]) + sq(fy - cy[So]));
    return tvd_usualy_d(st, cx, cy, fx, fy, Ms, Mx, My, So, Sd, m_has_axis, tracked, dM, dS, status);
}

// Gran::Get_par_TVD of an Axis face (Gran.cpp:486-519).
__device__ __forceinline__ St5 tvd_axis(const double* const* st, const double* cx, const double* cy, double fx,
                                        double fy, const St5& Ms, double Mx, double My, int Sd) {
    St5 o = Ms;
    if (Sd < 0) return o;  // no TVD partner: the upload rejects such a grid for the MK2 form
    const St5 par1 = load_state(st, Sd);
    const double dist2 = sqrt(sq(fx - Mx) + sq(fy - My));
    const double dist1 = sqrt(sq(fx - cx[Sd]) + sq(fy - cy[Sd]));
    o.v = linear3(-dist1, par1.v, -dist2, Ms.v, dist2, -Ms.v, 0.0);
    return o;
}

// Gran::Get_par_TVD_radial (Gran.cpp:562-675), ro and p only (the callers
// use no other field).  rp[c] = |centroid of c|^(2 gamma) is computed once
// per cell and step; pdis = |face centre|^(2 gamma) once per face (the
// reference evaluates pow at every use).
// r: |face centre|, r2 / r3: |centroid| of M / So, dM / dS: distances from
// the face centre to those centroids (computed by the face unit, passed in).
__device__ void tvd_radial_d(const double* const* st, const double* cx, const double* cy, const double* rp,
                             double fx, double fy, const St5& Ms, double Mx, double My, double rpM, int So, int Sd,
                             bool m_has_axis, double pdis, double r, double r2, double r3, double dM, double dS,
                             double& oro, double& op) {
    if (Sd < 0) {
        if (!m_has_axis) {
            oro = Ms.ro;
            op = Ms.p;
            return;
        }
        const St5 par3 = load_state(st, So);
        const double dist2 = dM;
        const double dist3 = dS;
        const double dist1 = sqrt(sq(fx - Mx) + sq(fy - (-My)));
        const double r12 = 1.0 / (-dist1 - (-dist2)), r23 = 1.0 / (-dist2 - dist3);
        // the mirrored centre has the radius of M itself
        oro = linear3r(Ms.ro * sq(r2), Ms.ro * sq(r2), par3.ro * sq(r3), r12, r23, -dist2) / sq(r);
        op = linear3r(Ms.p * rpM, Ms.p * rpM, par3.p * rp[So], r12, r23, -dist2) / pdis;
        return;
    }
    const St5 par1 = load_state(st, Sd);
    const St5 par3 = load_state(st, So);
    const double dist2 = dM;
    const double dist3 = dS;
    const double dx = cx[Sd], dy = cy[Sd];
    const double r1 = sqrt(sq(dx) + sq(dy));
    const double dist1 = sqrt(sq(fx - dx) + sq(fy - dy));
    const double r12 = 1.0 / (-dist1 - (-dist2)), r23 = 1.0 / (-dist2 - dist3);
    oro = linear3r(par1.ro * sq(r1), Ms.ro * sq(r2), par3.ro * sq(r3), r12, r23, -dist2) / sq(r);
    op = linear3r(par1.p * rp[Sd], Ms.p * rpM, par3.p * rp[So], r12, r23, -dist2) / pdis;
}
__device__ void tvd_radial(const double* const* st, const double* cx, const double* cy, const double* rp, double fx,
                           double fy, const St5& Ms, double Mx, double My, double rpM, int So, int Sd,
                           bool m_has_axis, double pdis, double& oro, double& op) {
    const double r = sqrt(sq(fx) + sq(fy));
    if (Sd < 0) {
        if (!m_has_axis) {
            oro = Ms.ro;
            op = Ms.p;
            return;
        }
        const St5 par3 = load_state(st, So);
        const double r2 = sqrt(sq(Mx) + sq(My));
        const double dist2 = sqrt(sq(fx - Mx) + sq(fy - My));
        const double sx = cx[So], sy = cy[So];
        const double r3 = sqrt(sq(sx) + sq(sy));
        const double dist3 = sqrt(sq(fx - sx) + sq(fy - sy));
        const double dist1 = sqrt(sq(fx - Mx) + sq(fy - (-My)));
        const double r12 = 1.0 / (-dist1 - (-dist2)), r23 = 1.0 / (-dist2 - dist3);
        // the mirrored centre has the radius of M itself
        oro = linear3r(Ms.ro * sq(r2), Ms.ro * sq(r2), par3.ro * sq(r3), r12, r23, -dist2) / sq(r);
        op = linear3r(Ms.p * rpM, Ms.p * rpM, par3.p * rp[So], r12, r23, -dist2) / pdis;
        return;
    }
    const St5 par1 = load_state(st, Sd);
    const St5 par3 = load_state(st, So);
    const double r2 = sqrt(sq(Mx) + sq(My));
    const double dist2 = sqrt(sq(fx - Mx) + sq(fy - My));
    const double sx = cx[So], sy = cy[So];
    const double r3 = sqrt(sq(sx) + sq(sy));
    const double dist3 = sqrt(sq(fx - sx) + sq(fy - sy));
    const double dx = cx[Sd], dy = cy[Sd];
    const double r1 = sqrt(sq(dx) + sq(dy));
    const double dist1 = sqrt(sq(fx - dx) + sq(fy - dy));
    const double r12 = 1.0 / (-dist1 - (-dist2)), r23 = 1.0 / (-dist2 - dist3);
    oro = linear3r(par1.ro * sq(r1), Ms.ro * sq(r2), par3.ro * sq(r3), r12, r23, -dist2) / sq(r);
    op = linear3r(par1.p * rp[Sd], Ms.p * rpM, par3.p * rp[So], r12, r23, -dist2) / pdis;
}

// Get_Sourse_MK1 (Cell.cpp:528-555): the pair of cells of k's radial chain
// whose r_istoch bracket the centroid radius rr (K_posle = Next(K_do)).
// Returns false (and raises ST_CHAIN) where the reference would follow a
// missing Back/Next link.
// `cached` (out): the cache entry read, so that the caller rewrites it only
// where the bracket changed.
__device__ bool source_bracket(const DevMesh& d, int k, double rr, int& K_do, int& K_posle, int* status,
                               int2* cached_out = nullptr) {
    K_do = d.cback[k];
    K_posle = d.cnext[k];
    const double ri = d.r_istoch[k];
    const int2 cpair = d.src_lo ? d.src_lo[k] : make_int2(-1, -1);
    if (cached_out) *cached_out = cpair;
    const int cached = cpair.x;
    if (cached >= 0) {
        // The reference walks the radial chain from the cell itself.  Along
        // a chain r_istoch increases strictly (checked at upload), so the
        // bracket it finds is unique: r[lo] <= rr < r[hi] when rr <
        // r_istoch, r[lo] < rr <= r[hi] otherwise, with hi = Next(lo).
        // Searching from last step's bracket finds the same pair in a step
        // or two.
        const bool caseA = rr < ri;
        {
            // the walk's first step, from the cached pair (hi = Next(lo)
            // cached too): both radii and the link the reference
            // dereferences are loaded together, one level of loads
            const int hi = cpair.y;
            const double rlo = d.r_istoch[cached], rhi = d.r_istoch[hi];
            const int link = caseA ? d.cback[cached] : d.cnext[hi];
            const bool below = caseA ? (rr < rlo) : !(rr > rlo);
            const bool above = caseA ? !(rr < rhi) : (rr > rhi);
            if (!below && !above) {
                if (link < 0) {
                    *status |= ST_CHAIN;
                    return false;
                }
                K_do = cached;
                K_posle = hi;
                return true;
            }
        }
        int lo = cached;
        int guard = 0;
        for (;;) {
            const int hi = d.cnext[lo];
            if (hi < 0 || ++guard > d.n_cells) {
                lo = -1;
                break;
            }
            const double rlo = d.r_istoch[lo], rhi = d.r_istoch[hi];
            const bool below = caseA ? (rr < rlo) : !(rr > rlo);
            const bool above = caseA ? !(rr < rhi) : (rr > rhi);
            if (below) {
                lo = d.cback[lo];
                if (lo < 0) break;
            } else if (above) {
                lo = hi;
            } else {
                break;
            }
        }
        // the reference dereferences Back of the lower cell (rr < r_istoch)
        // or Next of the upper cell (otherwise); a missing link is its crash
        if (lo < 0 || (caseA ? d.cback[lo] < 0 : d.cnext[d.cnext[lo]] < 0)) {
            *status |= ST_CHAIN;
            return false;
        }
        K_do = lo;
        K_posle = d.cnext[lo];
    } else if (rr < ri) {
        double r1 = ri;
        int guard = 0;
        while (r1 > rr) {
            if (K_do < 0 || ++guard > d.n_cells) {
                *status |= ST_CHAIN;
                return false;
            }
            r1 = d.r_istoch[K_do];
            K_do = d.cback[K_do];
        }
        if (K_do < 0) {
            *status |= ST_CHAIN;
            return false;
        }
        K_do = d.cnext[K_do];
        K_posle = K_do >= 0 ? d.cnext[K_do] : -1;
    } else {
        double r2 = ri;
        int guard = 0;
        while (r2 < rr) {
            if (K_posle < 0 || ++guard > d.n_cells) {
                *status |= ST_CHAIN;
                return false;
            }
            r2 = d.r_istoch[K_posle];
            K_posle = d.cnext[K_posle];
        }
        if (K_posle < 0) {
            *status |= ST_CHAIN;
            return false;
        }
        K_posle = d.cback[K_posle];
        K_do = K_posle >= 0 ? d.cback[K_posle] : -1;
    }
    if (K_do < 0 || K_posle < 0) {
        *status |= ST_CHAIN;
        return false;
    }
    return true;
}

// Monte-Carlo moments of species s seen by cell k (Cell.cpp:528-589): radial
// interpolation between the chain cells K_do and K_posle inside the source
// region, the cell's own moments outside it.  Also the k_u, k_v, k_T factors.
struct SrcMoments {
    double uH, vH, roH, pH, ku, kv, kT;
};
__device__ __forceinline__ SrcMoments source_moments(const DevMesh& d, int k, int s, bool interp, int K_do, int K_posle,
                                                     double rr, bool with_k = true) {
    SrcMoments m;
    if (interp) {
        const double r1 = d.r_istoch[K_do];
        const double r2 = d.r_istoch[K_posle];
        // linear(r1, t1, r2, t2, rr) with one reciprocal for all fields
        const double ir = 1.0 / (r1 - r2), dr = rr - r2;
        auto lin = [&](double t1, double t2) { return (t1 - t2) * ir * dr + t2; };
        m.uH = lin(d.Hu[4 * K_do + s], d.Hu[4 * K_posle + s]);
        m.vH = lin(d.Hv[4 * K_do + s], d.Hv[4 * K_posle + s]);
        m.roH = lin(d.Hn[4 * K_do + s], d.Hn[4 * K_posle + s]);
        const double TH = lin(d.HT[4 * K_do + s], d.HT[4 * K_posle + s]);
        m.ku = m.kv = m.kT = 0.0;
        if (with_k) {
            m.ku = lin(d.ku[K_do], d.ku[K_posle]);
            m.kv = lin(d.kv[K_do], d.kv[K_posle]);
            m.kT = lin(d.kT[K_do], d.kT[K_posle]);
        }
        m.pH = 0.5 * TH * m.roH;
    } else {
        m.uH = d.Hu[4 * k + s];
        m.vH = d.Hv[4 * k + s];
        m.roH = d.Hn[4 * k + s];
        m.pH = 0.5 * d.HT[4 * k + s] * d.Hn[4 * k + s];
        m.ku = with_k ? d.ku[k] : 0.0;
        m.kv = with_k ? d.kv[k] : 0.0;
        m.kT = with_k ? d.kT[k] : 0.0;
    }
    return m;
}

// Charge-exchange momentum / energy exchange rates of one species
// (Cell.cpp:590-660): nu_u, nu_v, nu_e before the sum over species.
__device__ __forceinline__ void source_rates(const gelios_params& P, SrcMoments m, double u, double v, double ro,
                                             double pro, double kin, double& nuu, double& nuv, double& nue) {
    if (m.roH <= 0.0) {
        m.roH = 0.0000001;
        m.pH = 0.0;
    }
    const double th = 2.0 * m.pH / m.roH;
    const double du2 = sq(u - m.uH) + sq(v - m.vH);
    const double UM = sqrt(du2 + (64.0 / (9.0 * kPi)) * (pro + th));
    const double UH = sqrt(du2 + (4.0 / kPi) * (pro + th));
    const double sig = sq(1.0 - P.a_2 * log(UM));
    const double nu = ro * m.roH * UM * sig;
    nuu = nu * (m.uH - u);
    nuv = nu * (m.vH - v);
    nue = nu * ((sq(m.uH) + sq(m.vH) - kin) / 2.0 + (UH / UM) * (th - pro));
}

// Get_Sourse_MK1 rates of one species from the temperature-like th = 2 pH / roH
// (Cell.cpp:590-660): one reciprocal square root serves |U_M|, U_H / U_M, and
// log U_M = log(U_M^2) / 2 waits for neither.
__device__ __forceinline__ void source_rates_th(const gelios_params& P, double uH, double vH, double roH, double th,
                                                double u, double v, double ro, double pro, double kin, double& nuu,
                                                double& nuv, double& nue) {
    const double du2 = sq(u - uH) + sq(v - vH), a = pro + th;
    const double UM2 = du2 + (64.0 / (9.0 * kPi)) * a, UH2 = du2 + (4.0 / kPi) * a;
    const double r = rsqrt(UM2);
    const double sig = sq(1.0 - P.a_2 * (0.5 * log(UM2)));
    const double nu = ro * roH * (UM2 * r) * sig;
    nuu = nu * (uH - u);
    nuv = nu * (vH - v);
    nue = nu * ((sq(uH) + sq(vH) - kin) / 2.0 + (sqrt(UH2) * r) * (th - pro));
}

// Cell::Get_Sourse_MK1 (Cell.cpp:498-665), one thread per cell.
__device__ void source_mk1(const DevMesh& d, const gelios_params& P, int k, double xx, double yy, double u, double v,
                           double ro, double p, double& q1, double& q2, double& q3, int* status) {
    const double rr = sqrt(sq(xx) + sq(yy));
    const bool interp = rr > P.src_rmin && rr < P.src_rmax && xx >= 0.0;
    int K_do = -1, K_posle = -1;
    if (interp) {
        if (!source_bracket(d, k, rr, K_do, K_posle, status)) {
            q1 = q2 = q3 = 0.0;
            return;
        }
        if (d.src_lo_out) d.src_lo_out[k] = make_int2(K_do, K_posle);
    }
    const double pro = p / ro;
    const double kin = sq(u) + sq(v);
    double nuu[4], nuv[4], nue[4];
    SrcMoments m;
#pragma unroll
    for (int s = 0; s < 4; s++) {
        m = source_moments(d, k, s, interp, K_do, K_posle, rr);
        source_rates(P, m, u, v, ro, pro, kin, nuu[s], nuv[s], nue[s]);
    }
    const double Mu = P.src_coef * (nuu[0] + nuu[1] + nuu[2] + nuu[3]);
    const double Mv = P.src_coef * (nuv[0] + nuv[1] + nuv[2] + nuv[3]);
    const double MT = P.src_coef * (nue[0] + nue[1] + nue[2] + nue[3]);
    q1 = Mu * m.ku;
    q2 = Mv * m.kv;
    q3 = MT * m.kT;
}

// The flux rows of the moving-grid forms hold each face unit's F.S once, as
// its owner sees it; the other side of an interior face takes its negative.
// w: the s_unit word of a cell's slot (unit << 1 | 1 on the other side).
__device__ __forceinline__ double unit_flux(const double* __restrict__ row, int w) {
    const double v = row[w >> 1];
    return (w & 1) ? -v : v;
}

// Block-level minimum of `t` (non-negative doubles; NaN ignored) folded into
// the device word acc with one atomicMin per block; clamp counters likewise.
__device__ __forceinline__ void block_reduce_commit(double t, int nro, int np_, int status, unsigned long long* acc,
                                                    unsigned long long* counters, int* status_word) {
    __shared__ double smin[32];
    __shared__ int sro[32], sp[32], sst[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ot = __shfl_down_sync(0xffffffffu, t, o);
        t = (ot < t) ? ot : t;
        nro += __shfl_down_sync(0xffffffffu, nro, o);
        np_ += __shfl_down_sync(0xffffffffu, np_, o);
        status |= __shfl_down_sync(0xffffffffu, status, o);
    }
    if (lane == 0) {
        smin[wid] = t;
        sro[wid] = nro;
        sp[wid] = np_;
        sst[wid] = status;
    }
    __syncthreads();
    if (wid == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        t = lane < nw ? smin[lane] : __longlong_as_double(0x7ff0000000000000LL);
        nro = lane < nw ? sro[lane] : 0;
        np_ = lane < nw ? sp[lane] : 0;
        status = lane < nw ? sst[lane] : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ot = __shfl_down_sync(0xffffffffu, t, o);
            t = (ot < t) ? ot : t;
            nro += __shfl_down_sync(0xffffffffu, nro, o);
            np_ += __shfl_down_sync(0xffffffffu, np_, o);
            status |= __shfl_down_sync(0xffffffffu, status, o);
        }
        if (lane == 0) {
            if (t >= 0.0 && t < __longlong_as_double(0x7ff0000000000000LL))
                atomicMin(acc, static_cast<unsigned long long>(__double_as_longlong(t)));
            if (nro) atomicAdd(&counters[0], static_cast<unsigned long long>(nro));
            if (np_) atomicAdd(&counters[1], static_cast<unsigned long long>(np_));
            if (status) atomicOr(status_word, status);
        }
    }
}

// ------------------------------------------------------------------ kernels
__global__ void centroid_kernel(DevMesh d, const double* __restrict__ X, const double* __restrict__ Y, double* cx,
                                double* cy, double* rp, double g2, double* vs, double* vol) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= d.n_cells) return;
    const int s = d.cstart[c], n = d.cstart[c + 1] - s;
    double x, y;
    centroid(d.contour + s, n, X, Y, x, y);
    cx[c] = x;
    cy[c] = y;
    rp[c] = pow2g(sqrt(sq(x) + sq(y)), g2);
    if (vs) {
        vs[c] = area(d.contour + s, n, d.sA, d.sB, d.gstart[c], d.gstart[c + 1], X, Y, false);
        vol[c] = volume_rotate(d.contour + s, n, X, Y);
    }
}

// ------------------------------------------------------------------ face units
// A face unit is one flux evaluation: an interior face (Usualy main face,
// evaluated once for both sides: the reference evaluates it from each side
// and the two results are the negatives of each other up to rounding,
// Setka.cpp:10195-10380) or a one-sided face (boundary types, evaluated for
// its owner only).  Each unit writes F*S once, into its own flux row, as the
// owner sees it (the neighbour's sum subtracts it; the plain form's two-phase
// kernels keep a row per slot and write -F*S into the twin's), and folds the
// CFL candidates of the sides whose cell is updated this step into the dt
// word.  The cell kernels then sum their slots in Grans order.

// ------------------------------------------------------------------ plain form, FP32 fluxes
// A change in the order or contraction of the operations around an FP32 flux
// moves its result by 1e-7 (an FP64 one by 1e-16), so this form keeps its
// kernels; the FP64 and FP32-wave-speed forms have their own below.
// Geometry of a face unit as its owner sees it: face centre (x2, y2), unit
// normal (n1, n2) for the end points in the owner's order, |centre|^2, the
// face length S, and the distances owner centroid - face centre and
// neighbour centroid - face centre (0 without a neighbour).  The same
// expressions as Setka.cpp:5244-5306 (t = B - A normalised, n = (t2, -t1));
// the twin's view has the normal negated and the two distances swapped.
struct FaceGeo {
    double x2, y2, n1, n2, f2, S, dist, distn;
};
__device__ __forceinline__ FaceGeo face_geo(double xa, double ya, double xb, double yb, double x, double y,
                                            bool has_nb, double x3, double y3) {
    FaceGeo f;
    f.x2 = (xa + xb) / 2.0;
    f.y2 = (ya + yb) / 2.0;
    double t1 = xb - xa, t2 = yb - ya;
    const double nn = sqrt(sq(t1) + sq(t2));
    f.S = nn;
    t1 = t1 / nn;
    t2 = t2 / nn;
    f.n1 = t2;
    f.n2 = -t1;
    f.f2 = sq(f.x2) + sq(f.y2);
    f.dist = sqrt(sq(x - f.x2) + sq(y - f.y2));
    f.distn = has_nb ? sqrt(sq(x3 - f.x2) + sq(y3 - f.y2)) : 0.0;
    return f;
}

// Go_stationary flux of one side (Setka.cpp:5244-5306): owner state `own`
// at centre (x, y), radius rad; face centre (x2, y2), normal (n1, n2) and
// |centre|^2 f2 as seen from the owner; neighbour (for Usualy faces)
// state, centre and radius rad_nb.  pfc: |face centre|^(2 gamma) if cached,
// else negative.
template <typename TF>
__device__ __forceinline__ double stationary_side(const gelios_params& P, int ft, const St5& own, double x, double y,
                                                  double rad, double rpo, double x2, double y2, double n1, double n2,
                                                  double f2, const St5& nbs, double x3, double y3, double rad_nb,
                                                  double rpn, double pfc, FluxOut<double>& F) {
    const double g2 = 2 * P.gamma;
    St5 par11 = own;
    St5 par2 = own;
    if (ft == G_USUALY) par2 = nbs;
    else if (ft == G_EXTERN) {
        if (par2.u >= 0.0) par2.u = P.extern_u_par;
    } else if (ft == G_AXIS) par2.v = -par2.v;
    else if (ft == G_INNER_SPHERE) par2 = inner_sphere_state(P, x2, y2);
    else if (ft == G_INPUT) par2 = input_state(P);
    if (rad < P.rad_stat && ft == G_USUALY) {
        const double pf = pfc >= 0.0 ? pfc : pow2g(sqrt(f2), g2);  // (rad/fr)^(2g) = rad^(2g) / fr^(2g)
        par11.ro = par11.ro * sq(rad) / f2;
        par2.ro = par2.ro * sq(rad_nb) / f2;
        par11.p = par11.p * (rpo / pf);
        par2.p = par2.p * (rpn / pf);
        polar_perenos(x, y, x2, y2, par11.u, par11.v);
        polar_perenos(x3, y3, x2, y2, par2.u, par2.v);
    } else if (ft == G_INNER_SPHERE) {
        par11.ro = par11.ro * sq(rad) / f2;
        par11.p = par11.p * (rpo / (pfc >= 0.0 ? pfc : pow2g(sqrt(f2), g2)));
    } else if (rad < P.rad_stat && ft == G_AXIS) {
        polar_perenos(x, y, x2, y2, par11.u, par11.v);
        par11.v = 0.0;
        par2 = par11;
    } else if (ft == G_AXIS) {
        par11.v = 0.0;
        par2 = par11;
    }
    return hllc_flux<TF>(P.gamma, P.kurant, par11, par2, 0.0, n1, n2, 1.0, 1, false, F);  // UU
}

// One Go_stationary face unit: slot fluxes of the owner (and of the twin)
// and the minimum of its CFL candidates (+inf if none).  Inlined into the
// per-step kernel and into the cooperative multi-step kernel; the two
// compilations may contract multiply-adds differently (last-bit
// differences, a non-inlined body costs 12% per step).
template <typename TF>
__device__ __forceinline__ double stationary32_unit_body(const DevMesh& d, const gelios_params& P, const StepBuffers& b,
                                                       double* __restrict__ fl, int u) {
    double tmin_u = __longlong_as_double(0x7ff0000000000000LL);
    const size_t ng = d.n_slots;
    {
        const int g = d.u_slot[u], K = d.u_cell[u], gt = d.u_twin[u];
        const bool procK = !(d.cflags[K] & CF_CENTR);
        const int nb = gt >= 0 ? d.snb[g] : -1;
        const bool procN = nb >= 0 && !(d.cflags[nb] & CF_CENTR);
        if (procK || procN) {
            const int ft = d.sinfo[g] & SI_TYPE_MASK;
            const double x = b.cx[K], y = b.cy[K];
            const double rad = sqrt(sq(x) + sq(y));
            const St5 own = load_state(b.cur, K);
            St5 nbs = own;
            double x3 = 0.0, y3 = 0.0, radn = 0.0;
            if (nb >= 0) {
                nbs = load_state(b.cur, nb);
                x3 = b.cx[nb];
                y3 = b.cy[nb];
                radn = sqrt(sq(x3) + sq(y3));
            }
            FaceGeo f;
            if (b.fgeo) {
                const size_t nu = d.n_units;
                f.x2 = b.fgeo[u];
                f.y2 = b.fgeo[nu + u];
                f.n1 = b.fgeo[2 * nu + u];
                f.n2 = b.fgeo[3 * nu + u];
                f.f2 = b.fgeo[4 * nu + u];
                f.S = b.fgeo[5 * nu + u];
                f.dist = b.fgeo[6 * nu + u];
                f.distn = b.fgeo[7 * nu + u];
            } else {
                const int A = d.sA[g], B = d.sB[g];
                f = face_geo(d.X[A], d.Y[A], d.X[B], d.Y[B], x, y, nb >= 0, x3, y3);
            }
            const double S = f.S;
            FluxOut<double> F;
            const double rpK = b.rp[K], rpN = nb >= 0 ? b.rp[nb] : 0.0;
            const double pfc = b.upf ? b.upf[u] : -1.0;
            const double UU = stationary_side<TF>(P, ft, own, x, y, rad, rpK, f.x2, f.y2, f.n1, f.n2, f.f2, nbs, x3,
                                                  y3, radn, rpN, pfc, F);
            fl[0 * ng + g] = F.P0 * S;
            fl[1 * ng + g] = F.P1 * S;
            fl[2 * ng + g] = F.P2 * S;
            fl[3 * ng + g] = F.P3 * S;
            fl[4 * ng + g] = F.PQ * S;
            if (procK) tmin_u = dmin_ref(tmin_u, P.kurant * f.dist / UU);
            if (gt >= 0) {
                // the twin's evaluation mirrors this one unless the radial
                // scaling switches at rad_stat between the two cells
                const bool same = (rad < P.rad_stat) == (radn < P.rad_stat);
                if (same) {
                    fl[0 * ng + gt] = -(F.P0 * S);
                    fl[1 * ng + gt] = -(F.P1 * S);
                    fl[2 * ng + gt] = -(F.P2 * S);
                    fl[3 * ng + gt] = -(F.P3 * S);
                    fl[4 * ng + gt] = -(F.PQ * S);
                    if (procN) tmin_u = dmin_ref(tmin_u, P.kurant * f.distn / UU);
                } else {
                    FluxOut<double> G;
                    const double Un = stationary_side<TF>(P, ft, nbs, x3, y3, radn, rpN, f.x2, f.y2, -f.n1, -f.n2,
                                                          f.f2, own, x, y, rad, rpK, pfc, G);
                    fl[0 * ng + gt] = G.P0 * S;
                    fl[1 * ng + gt] = G.P1 * S;
                    fl[2 * ng + gt] = G.P2 * S;
                    fl[3 * ng + gt] = G.P3 * S;
                    fl[4 * ng + gt] = G.PQ * S;
                    if (procN) tmin_u = dmin_ref(tmin_u, P.kurant * f.distn / Un);
                }
            }
        }
    }
    return tmin_u;
}

template <typename TF>
__global__ void __launch_bounds__(128) stationary32_unit_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                              double* __restrict__ fl) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    double tmin_u = __longlong_as_double(0x7ff0000000000000LL);
    if (u < d.n_units) tmin_u = stationary32_unit_body<TF>(d, P, b, fl, u);
    block_reduce_commit(tmin_u, 0, 0, 0, b.dt_acc, b.counters, b.status);
}

// Go_stationary cell update (Setka.cpp:5309-5341) of cell c from the summed
// slots; folds its `time` mark and clamps into tmark, nro, npc.
__device__ __forceinline__ void stationary32_update_body(const DevMesh& d, const gelios_params& P, const StepBuffers& b,
                                                       const double* __restrict__ fl, int c, double& tmark, int& nro,
                                                       int& npc) {
    const size_t ng = d.n_slots;
    if (!(d.cflags[c] & CF_CENTR)) {
        tmark = dmin_ref(tmark, 10000000.0);  // `time` starts at 1e7 in every step (Setka.cpp:5222)
        const double dt = *b.dt_cur;
        const St5 par1 = load_state(b.cur, c);
        const double y = b.cy[c];
        const int g0 = d.gstart[c], g1 = d.gstart[c + 1];
        double Pt0 = 0.0, Pt1 = 0.0, Pt2 = 0.0, Pt3 = 0.0, Pt4 = 0.0;
        for (int g = g0; g < g1; g++) {
            Pt0 = Pt0 + fl[0 * ng + g];
            Pt1 = Pt1 + fl[1 * ng + g];
            Pt2 = Pt2 + fl[2 * ng + g];
            Pt3 = Pt3 + fl[3 * ng + g];
            Pt4 = Pt4 + fl[4 * ng + g];
        }
        // the cell's area: cached with the centroids (the plain grid does not
        // move), or computed here when no cache is given
        double Volume;
        if (b.vs) {
            Volume = b.vs[c];
        } else {
            const int s0 = d.cstart[c], n = d.cstart[c + 1] - s0;
            Volume = area(d.contour + s0, n, d.sA, d.sB, g0, g1, d.X, d.Y, false);
        }
        const double gm1 = P.gamma - 1;
        double ro3 = par1.ro - dt * (Pt0 / Volume + par1.ro * par1.v / y);
        const double Q33 = par1.Q - (dt / Volume) * Pt4 - dt * par1.Q * par1.v / y;
        if (ro3 <= 0) {
            ro3 = P.ro_floor;
            nro++;
        }
        const double uu = par1.u * par1.u + par1.v * par1.v;
        const double u3 = (par1.ro * par1.u - dt * (Pt1 / Volume + par1.ro * par1.v * par1.u / y)) / ro3;
        const double v3 = (par1.ro * par1.v - dt * (Pt2 / Volume + par1.ro * par1.v * par1.v / y)) / ro3;
        double p3 = (((par1.p / gm1 + par1.ro * uu * 0.5) -
                      dt * (Pt3 / Volume + par1.v * (P.gamma * par1.p / gm1 + par1.ro * uu * 0.5) / y)) -
                     0.5 * ro3 * (u3 * u3 + v3 * v3)) *
                    gm1;
        if (p3 <= 0) {
            p3 = P.p_floor;
            npc++;
        }
        b.nxt[0][c] = ro3;
        b.nxt[1][c] = p3;
        b.nxt[2][c] = u3;
        b.nxt[3][c] = v3;
        b.nxt[4][c] = Q33;
    }
}

__global__ void __launch_bounds__(128) stationary32_update_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                                const double* __restrict__ fl) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    double tmark = __longlong_as_double(0x7ff0000000000000LL);
    int nro = 0, npc = 0;
    if (c < d.n_cells) stationary32_update_body(d, P, b, fl, c, tmark, nro, npc);
    block_reduce_commit(tmark, nro, npc, 0, b.dt_acc, b.counters, b.status);
}

// `nsteps` Go_stationary steps in one cooperative launch: every block
// strides over the face units, then (grid barrier) over the cells, then
// (barrier) one thread turns the CFL minimum into the next step's dt
// (barrier).  The same unit and cell bodies as the three-kernel path; the
// grid is sized to be fully resident (cooperative launch).  21 us per step
// against 29 us for three launches per step on the 180 x 120 grid.
// bs[0] / bs[1]: the buffers of even / odd steps.
template <typename TF>
__global__ void __launch_bounds__(128) stationary32_persistent_kernel(DevMesh d, gelios_params P, StepBuffers b0,
                                                                    StepBuffers b1, double* __restrict__ fl,
                                                                    int nsteps) {
    cg::grid_group grid = cg::this_grid();
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nth = gridDim.x * blockDim.x;
    for (int st = 0; st < nsteps; st++) {
        const StepBuffers& b = (st & 1) ? b1 : b0;
        double tmin = __longlong_as_double(0x7ff0000000000000LL);
        for (int u = tid; u < d.n_units; u += nth) tmin = dmin_ref(tmin, stationary32_unit_body<TF>(d, P, b, fl, u));
        block_reduce_commit(tmin, 0, 0, 0, b.dt_acc, b.counters, b.status);
        grid.sync();
        double tmark = __longlong_as_double(0x7ff0000000000000LL);
        int nro = 0, npc = 0;
        for (int c = tid; c < d.n_cells; c += nth) stationary32_update_body(d, P, b, fl, c, tmark, nro, npc);
        block_reduce_commit(tmark, nro, npc, 0, b.dt_acc, b.counters, b.status);
        grid.sync();
        if (tid == 0) {
            const unsigned long long a = *b.dt_acc;
            *b.dt_next = (a == 0x7ff0000000000000ULL) ? 100000000.0 : __longlong_as_double(static_cast<long long>(a));
            *b.dt_acc = 0x7ff0000000000000ULL;
        }
        grid.sync();
    }
}

// `nsteps` Go_stationary steps of many instances in one cooperative launch.
// The instances share the mesh (topology and geometry) and have their own
// parameters (inflow and inner-wind states), state buffers, flux slots and
// dt words.  Work is dealt in 128-wide tiles of one instance each, so every
// block folds its CFL minimum into one instance's dt word; after the cell
// phase one thread per instance turns its minimum into the next dt.  The
// unit and cell bodies are the one-instance kernels'.  `active` lists the
// instances advanced by this launch (the others keep their state).
template <typename TF>
__global__ void __launch_bounds__(128) stationary32_batch_kernel(DevMesh d, const PlainInstance* __restrict__ inst,
                                                               const int* __restrict__ active, int n_active,
                                                               int nsteps) {
    cg::grid_group grid = cg::this_grid();
    const int ut = (d.n_units + 127) / 128, ct = (d.n_cells + 127) / 128;
    for (int st = 0; st < nsteps; st++) {
        const int par = st & 1;
        for (int t = blockIdx.x; t < n_active * ut; t += gridDim.x) {
            const PlainInstance& I = inst[active[t / ut]];
            const int u = (t % ut) * 128 + threadIdx.x;
            double tmin = __longlong_as_double(0x7ff0000000000000LL);
            if (u < d.n_units) tmin = stationary32_unit_body<TF>(d, I.P, I.b[par], I.fl, u);
            __syncthreads();  // the previous tile's reduction has read its shared words
            block_reduce_commit(tmin, 0, 0, 0, I.b[par].dt_acc, I.b[par].counters, I.b[par].status);
        }
        grid.sync();
        for (int t = blockIdx.x; t < n_active * ct; t += gridDim.x) {
            const PlainInstance& I = inst[active[t / ct]];
            const int c = (t % ct) * 128 + threadIdx.x;
            double tmark = __longlong_as_double(0x7ff0000000000000LL);
            int nro = 0, npc = 0;
            if (c < d.n_cells) stationary32_update_body(d, I.P, I.b[par], I.fl, c, tmark, nro, npc);
            __syncthreads();
            block_reduce_commit(tmark, nro, npc, 0, I.b[par].dt_acc, I.b[par].counters, I.b[par].status);
        }
        grid.sync();
        for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n_active; k += gridDim.x * blockDim.x) {
            const StepBuffers& b = inst[active[k]].b[par];
            const unsigned long long a = *b.dt_acc;
            *b.dt_next = (a == 0x7ff0000000000000ULL) ? 100000000.0 : __longlong_as_double(static_cast<long long>(a));
            *b.dt_acc = 0x7ff0000000000000ULL;
        }
        grid.sync();
    }
}

// ------------------------------------------------------------------ plain form
// What a face unit of the plain form reads of the (fixed) grid: unit normal
// (n1, n2) for the end points in the owner's order, length S, the distances
// owner centroid - face centre and neighbour centroid - face centre, and per
// side the radial scaling of Setka.cpp:5256-5290: kro = |centroid|^2 /
// |centre|^2, kp = (|centroid| / |centre|)^(2 gamma), and the rotation (C, S)
// from the polar frame of the centroid to that of the face centre
// (polar_perenos).  flags: bit 0 the owner's evaluation is scaled (centroid
// radius below rad_stat), bit 1 the neighbour's.  Inner-sphere faces hold
// |centre| and the centre in kroN, CN, SN.
struct UnitGeo {
    double n1, n2, S, dist, distn, kroO, kpO, CO, SO, kroN, kpN, CN, SN;
    uint32_t flags;
};
__device__ __forceinline__ UnitGeo unit_geo(double gamma, double rad_stat, int ft, double xa, double ya, double xb,
                                            double yb, int K, int nb, const double* cx, const double* cy,
                                            const double* rp) {
    UnitGeo f;
    const double x2 = (xa + xb) / 2.0, y2 = (ya + yb) / 2.0;
    double t1 = xb - xa, t2 = yb - ya;  // t = B - A normalised, n = (t2, -t1): Setka.cpp:5244-5306
    f.S = sqrt(sq(t1) + sq(t2));
    t1 = t1 / f.S;
    t2 = t2 / f.S;
    f.n1 = t2;
    f.n2 = -t1;
    const double f2 = sq(x2) + sq(y2), pf = pow2g(sqrt(f2), 2 * gamma);
    double cf, sf;
    polar_cs(x2, y2, cf, sf);
    auto side = [&](int c, double& dist, double& kro, double& kp, double& C, double& Sn) {
        const double x = cx[c], y = cy[c];
        dist = sqrt(sq(x - x2) + sq(y - y2));
        kro = (sq(x) + sq(y)) / f2;
        kp = rp[c] / pf;
        double c1, s1;
        polar_cs(x, y, c1, s1);
        C = c1 * cf + s1 * sf;
        Sn = c1 * sf - s1 * cf;
        return sqrt(sq(x) + sq(y)) < rad_stat;
    };
    f.flags = side(K, f.dist, f.kroO, f.kpO, f.CO, f.SO) ? 1u : 0u;
    f.distn = f.kroN = f.kpN = f.CN = f.SN = 0.0;
    if (nb >= 0) {
        f.flags |= side(nb, f.distn, f.kroN, f.kpN, f.CN, f.SN) ? 2u : 0u;
    } else if (ft == G_INNER_SPHERE) {
        f.kroN = sqrt(f2);
        f.CN = x2;
        f.SN = y2;
    }
    return f;
}

// Radial scaling and rotation of one side's state to the face centre.
__device__ __forceinline__ St5 plain_scale(const St5& s, double kro, double kp, double C, double Sn) {
    St5 o = s;
    o.ro = mul_rn(s.ro, kro);
    o.p = mul_rn(s.p, kp);
    o.u = fma_rn(s.u, C, -mul_rn(s.v, Sn));
    o.v = fma_rn(s.u, Sn, mul_rn(s.v, C));
    return o;
}
// Inner-sphere state from |centre| and the centre (inner_sphere_state without
// a sum, so that its bits do not depend on where it is inlined).
__device__ __forceinline__ St5 plain_inner_state(const gelios_params& P, double dist, double x, double y) {
    St5 s;
    s.ro = 1.0 / (P.chi * P.chi * dist * dist);
    s.p = s.ro * P.chi * P.chi / (P.gamma * P.inner_mach * P.inner_mach);
    s.u = P.chi * x / dist;
    s.v = P.chi * y / dist;
    s.Q = s.ro;
    return s;
}
// The two states of a boundary face as its owner sees it (Setka.cpp:5244-5306).
__device__ __forceinline__ void plain_boundary(const gelios_params& P, int ft, const St5& own, bool scaled,
                                               const UnitGeo& f, St5& L, St5& R) {
    L = own;
    R = own;
    if (ft == G_INNER_SPHERE) {
        L.ro = mul_rn(own.ro, f.kroO);
        L.p = mul_rn(own.p, f.kpO);
        R = plain_inner_state(P, f.kroN, f.CN, f.SN);
    } else if (ft == G_INPUT) {
        R = input_state(P);
    } else if (ft == G_EXTERN) {
        if (R.u >= 0.0) R.u = P.extern_u_par;
    } else if (ft == G_AXIS) {
        if (scaled) L.u = fma_rn(own.u, f.CO, -mul_rn(own.v, f.SO));
        L.v = 0.0;
        R = L;
    }
}

// One Go_stationary face unit: slot fluxes of the owner (and of the twin)
// and the minimum of its CFL candidates (+inf if none).
template <typename TF>
__device__ __forceinline__ double stationary_unit_body(const DevMesh& d, const gelios_params& P, const StepBuffers& b,
                                                       double* __restrict__ fl, int u) {
    double tmin_u = __longlong_as_double(0x7ff0000000000000LL);
    const size_t ng = d.n_slots;
    const int g = d.u_slot[u], K = d.u_cell[u], gt = d.u_twin[u];
    // the unit-major copies of the neighbour and the flags save a level of
    // dependent loads; the allocation-free entry has only the slots'
    int nb;
    uint32_t info, cfK, cfN;
    if (d.u_info) {
        nb = d.u_nb[u];
        info = d.u_info[u];
        cfK = info >> UI_CF_OWN;
        cfN = info >> UI_CF_NB;
    } else {
        nb = gt >= 0 ? d.snb[g] : -1;
        info = d.sinfo[g];
        cfK = d.cflags[K];
        cfN = nb >= 0 ? d.cflags[nb] : 0u;
    }
    const bool procK = !(cfK & CF_CENTR);
    const bool procN = nb >= 0 && !(cfN & CF_CENTR);
    if (!(procK || procN)) return tmin_u;
    const int ft = info & SI_TYPE_MASK;
    const St5 own = load_state(b.cur, K);
    St5 nbs = own;
    if (nb >= 0) nbs = load_state(b.cur, nb);
    UnitGeo f;
    if (b.ugeo) {
        const size_t nu = d.n_units;
        const double* r = b.ugeo + u;
        f.flags = reinterpret_cast<const uint32_t*>(b.ugeo + kUnitGeoRows * nu)[u];
        f.n1 = r[0];
        f.n2 = r[nu];
        f.S = r[2 * nu];
        f.dist = r[3 * nu];
        f.distn = r[4 * nu];
        if (f.flags || ft != G_USUALY) {
            f.kroO = r[5 * nu];
            f.kpO = r[6 * nu];
            f.CO = r[7 * nu];
            f.SO = r[8 * nu];
            f.kroN = r[9 * nu];
            f.kpN = r[10 * nu];
            f.CN = r[11 * nu];
            f.SN = r[12 * nu];
        }
    } else {
        const int A = d.sA[g], B = d.sB[g];
        f = unit_geo(P.gamma, P.rad_stat, ft, d.X[A], d.Y[A], d.X[B], d.Y[B], K, nb, b.cx, b.cy, b.rp);
    }
    double F[5];
    if (ft != G_USUALY) {
        St5 L, R;
        plain_boundary(P, ft, own, f.flags & 1u, f, L, R);
        const double UU = plain_flux<TF>(P, L, R, f.n1, f.n2, F);
#pragma unroll
        for (int k = 0; k < 5; k++) fl[k * ng + g] = mul_rn(F[k], f.S);
        return procK ? dmin_ref(tmin_u, mul_rn(P.kurant, f.dist) / UU) : tmin_u;
    }
    St5 L = own, R = nbs;
    if (f.flags & 1u) {
        L = plain_scale(own, f.kroO, f.kpO, f.CO, f.SO);
        R = plain_scale(nbs, f.kroN, f.kpN, f.CN, f.SN);
    }
    double UU = plain_flux<TF>(P, L, R, f.n1, f.n2, F);
#pragma unroll
    for (int k = 0; k < 5; k++) fl[k * ng + g] = mul_rn(F[k], f.S);
    // CFL candidates; a NaN one is none, as the reference's std::min leaves it
    if (procK) tmin_u = dmin_ref(tmin_u, mul_rn(P.kurant, f.dist) / UU);
    if (gt < 0) return tmin_u;
    double sg = -f.S;
    // the twin's evaluation mirrors this one unless the radial scaling
    // switches at rad_stat between the two cells
    if (f.flags == 1u || f.flags == 2u) {
        L = nbs;
        R = own;
        if (f.flags & 2u) {
            L = plain_scale(nbs, f.kroN, f.kpN, f.CN, f.SN);
            R = plain_scale(own, f.kroO, f.kpO, f.CO, f.SO);
        }
        UU = plain_flux<TF>(P, L, R, -f.n1, -f.n2, F);
        sg = f.S;
    }
#pragma unroll
    for (int k = 0; k < 5; k++) fl[k * ng + gt] = mul_rn(F[k], sg);
    if (procN) tmin_u = dmin_ref(tmin_u, mul_rn(P.kurant, f.distn) / UU);
    return tmin_u;
}

template <typename TF>
__global__ void __launch_bounds__(128) stationary_unit_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                              double* __restrict__ fl) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    double tmin_u = __longlong_as_double(0x7ff0000000000000LL);
    if (u < d.n_units) tmin_u = stationary_unit_body<TF>(d, P, b, fl, u);
    block_reduce_commit(tmin_u, 0, 0, 0, b.dt_acc, b.counters, b.status);
}

// Go_stationary update (Setka.cpp:5309-5341) of a cell from its summed
// fluxes; rV, ry: reciprocals of its area and of its centroid's y.
__device__ __forceinline__ St5 plain_update(const gelios_params& P, const St5& s, const double (&Pt)[5], double dt,
                                            double rV, double ry, int& nro, int& npc) {
    const double gm1 = P.gamma - 1, rg1 = 1.0 / gm1, ndt = -dt;
    const double roy = mul_rn(mul_rn(s.ro, s.v), ry);
    St5 o;
    o.ro = fma_rn(ndt, fma_rn(Pt[0], rV, roy), s.ro);
    o.Q = fma_rn(ndt, fma_rn(Pt[4], rV, mul_rn(mul_rn(s.Q, s.v), ry)), s.Q);
    if (o.ro <= 0) {
        o.ro = P.ro_floor;
        nro++;
    }
    const double rro = 1.0 / o.ro;
    o.u = mul_rn(fma_rn(ndt, fma_rn(Pt[1], rV, mul_rn(roy, s.u)), mul_rn(s.ro, s.u)), rro);
    o.v = mul_rn(fma_rn(ndt, fma_rn(Pt[2], rV, mul_rn(roy, s.v)), mul_rn(s.ro, s.v)), rro);
    const double ek = mul_rn(mul_rn(0.5, s.ro), fma_rn(s.u, s.u, mul_rn(s.v, s.v)));
    const double E = fma_rn(s.p, rg1, ek), H = fma_rn(mul_rn(P.gamma, s.p), rg1, ek);
    const double E3 = fma_rn(ndt, fma_rn(Pt[3], rV, mul_rn(mul_rn(s.v, H), ry)), E);
    o.p = mul_rn(sub_rn(E3, mul_rn(mul_rn(0.5, o.ro), fma_rn(o.u, o.u, mul_rn(o.v, o.v)))), gm1);
    if (o.p <= 0) {
        o.p = P.p_floor;
        npc++;
    }
    return o;
}

// The update of cell c from its slots; folds its `time` mark and clamps into
// tmark, nro, npc.
__device__ __forceinline__ void stationary_update_body(const DevMesh& d, const gelios_params& P, const StepBuffers& b,
                                                       const double* __restrict__ fl, int c, double dt, double& tmark,
                                                       int& nro, int& npc) {
    const size_t ng = d.n_slots;
    if (!(d.cflags[c] & CF_CENTR)) {
        tmark = dmin_ref(tmark, 10000000.0);  // `time` starts at 1e7 in every step (Setka.cpp:5222)
        const St5 par1 = load_state(b.cur, c);
        const double y = b.cy[c];
        const int g0 = d.gstart[c], g1 = d.gstart[c + 1];
        double Pt[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        if (g1 - g0 == 4) {  // quadrilaterals: all slot loads in flight together
            double a[5][4];
#pragma unroll
            for (int k = 0; k < 5; k++)
#pragma unroll
                for (int j = 0; j < 4; j++) a[k][j] = fl[k * ng + g0 + j];
#pragma unroll
            for (int k = 0; k < 5; k++) Pt[k] = (((Pt[k] + a[k][0]) + a[k][1]) + a[k][2]) + a[k][3];
        } else {
            for (int g = g0; g < g1; g++)
#pragma unroll
                for (int k = 0; k < 5; k++) Pt[k] = Pt[k] + fl[k * ng + g];
        }
        // the cell's area: cached with the centroids (the plain grid does not
        // move), or computed here when no cache is given
        double Volume;
        if (b.vs) {
            Volume = b.vs[c];
        } else {
            const int s0 = d.cstart[c], n = d.cstart[c + 1] - s0;
            Volume = area(d.contour + s0, n, d.sA, d.sB, g0, g1, d.X, d.Y, false);
        }
        const St5 o = plain_update(P, par1, Pt, dt, 1.0 / Volume, 1.0 / y, nro, npc);
        b.nxt[0][c] = o.ro;
        b.nxt[1][c] = o.p;
        b.nxt[2][c] = o.u;
        b.nxt[3][c] = o.v;
        b.nxt[4][c] = o.Q;
    }
}

__global__ void __launch_bounds__(128) stationary_update_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                                const double* __restrict__ fl) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    double tmark = __longlong_as_double(0x7ff0000000000000LL);
    int nro = 0, npc = 0;
    if (c < d.n_cells) stationary_update_body(d, P, b, fl, c, *b.dt_cur, tmark, nro, npc);
    block_reduce_commit(tmark, nro, npc, 0, b.dt_acc, b.counters, b.status);
}

// Minimum over a warp / block of doubles that are not NaN and not negative.
// Such doubles order as their bit patterns: two 32-bit warp reductions.
// The block's minimum is valid in every lane of warp 0; sm: a word per warp.
__device__ __forceinline__ double warp_min_nonneg(double t) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(t)), lo = static_cast<unsigned>(__double2loint(t));
    const unsigned mh = __reduce_min_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_min_sync(0xffffffffu, hi == mh ? lo : 0xffffffffu);
    return __hiloint2double(static_cast<int>(mh), static_cast<int>(ml));
}
__device__ __forceinline__ double block_min_nonneg(double t, double* sm) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    t = warp_min_nonneg(t);
    if (lane == 0) sm[wid] = t;
    __syncthreads();
    if (wid == 0) t = warp_min_nonneg(lane < nw ? sm[lane] : __longlong_as_double(0x7ff0000000000000LL));
    return t;
}
// CFL candidates in [0, inf): a NaN or negative one (a failed state) is none,
// as block_reduce_commit has it for a block's minimum.
__device__ __forceinline__ double dt_candidate(double t) {
    return t >= 0.0 ? t : __longlong_as_double(0x7ff0000000000000LL);
}
// The CFL accumulator of step st of a one-launch call: three in turn, each
// read after the step's grid barrier and re-armed a step later, when no block
// can still be reading it (words_init_kernel arms them at the start).
__device__ __forceinline__ unsigned long long* plain_acc(unsigned long long* acc, int st) {
    const int k = st % 3;
    return acc + (k ? 3 + k : 0);
}
// T[now2]: the accumulated minimum, 1e8 where no cell took part
__device__ __forceinline__ double plain_dt(unsigned long long a) {
    return (a == 0x7ff0000000000000ULL) ? 100000000.0 : __longlong_as_double(static_cast<long long>(a));
}

// `nsteps` Go_stationary steps in one cooperative launch: every block
// strides over the face units, then (grid barrier) over the cells (barrier).
// The CFL minimum of a step is complete at its first barrier, where every
// block reads the next dt.  Taken by grids that stationary_lanes_kernel does
// not hold.  b0 / b1: the buffers of even / odd steps.
template <typename TF>
__global__ void __launch_bounds__(128) stationary_persistent_kernel(DevMesh d, gelios_params P, StepBuffers b0,
                                                                    StepBuffers b1, double* __restrict__ fl,
                                                                    int nsteps) {
    __shared__ double sm[32];
    cg::grid_group grid = cg::this_grid();
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nth = gridDim.x * blockDim.x;
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    double dt = *b0.dt_cur, dt_prev = dt, tmark = inf;
    int nro = 0, npc = 0;
    // `time` starts at 1e7 in every step (Setka.cpp:5222) with a cell to update
    bool any = false;
    for (int c = tid; c < d.n_cells; c += nth) any |= !(d.cflags[c] & CF_CENTR);
    for (int st = 0; st < nsteps; st++) {
        const StepBuffers& b = (st & 1) ? b1 : b0;
        double t = any ? 10000000.0 : inf;
        for (int u = tid; u < d.n_units; u += nth)
            t = dmin_ref(t, dt_candidate(stationary_unit_body<TF>(d, P, b, fl, u)));
        unsigned long long* acc = plain_acc(b0.dt_acc, st);
        t = block_min_nonneg(t, sm);
        if (threadIdx.x == 0 && t < inf) atomicMin(acc, static_cast<unsigned long long>(__double_as_longlong(t)));
        grid.sync();
        const unsigned long long a = __ldcg(acc);
        if (tid == 0) *plain_acc(b0.dt_acc, st + 2) = 0x7ff0000000000000ULL;
        for (int c = tid; c < d.n_cells; c += nth) stationary_update_body(d, P, b, fl, c, dt, tmark, nro, npc);
        dt_prev = dt;
        dt = plain_dt(a);
        grid.sync();
    }
    if (nro) atomicAdd(&b0.counters[0], static_cast<unsigned long long>(nro));
    if (npc) atomicAdd(&b0.counters[1], static_cast<unsigned long long>(npc));
    if (tid == 0) {
        const StepBuffers& b = ((nsteps - 1) & 1) ? b1 : b0;
        *b.dt_next = dt;
        *const_cast<double*>(b.dt_cur) = dt_prev;
    }
}

// The same with four lanes per cell, one per face, for grids whose 4 n_cells
// lanes are resident at once and whose updated cells have at most four faces
// (plain_lane_threads).  What a face needs of the fixed grid is read once per
// call and stays in the lane's registers, as does the cell's own state; a
// step loads the neighbour's five values, evaluates the face, adds the four
// fluxes in Grans order by shuffles and updates the cell: no flux slots and
// ONE grid barrier per step.  An interior face is evaluated by both its
// cells with the same operands (in the main face's orientation), so the
// results are those of the two-phase kernel.
// Bound by latency (the gather from L2, the chain of the HLLC flux, the
// barrier).  180 x 120 cells: 18.2 us per step in two phases with three grid
// barriers, 5.0 us here; 77 x 45 cells: 17.3 and 3.9 us.
constexpr int kLaneThreads = 640;
template <typename TF>
__global__ void __launch_bounds__(kLaneThreads, 1) stationary_lanes_kernel(DevMesh d, gelios_params P, StepBuffers b0,
                                                                           StepBuffers b1, int nsteps) {
    __shared__ double sm[32];
    cg::grid_group grid = cg::this_grid();
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = tid >> 2, j = tid & 3, q0 = threadIdx.x & 28;
    const unsigned full = 0xffffffffu;
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    const bool act = c < d.n_cells && !(d.cflags[c] & CF_CENTR);
    double ry = 0.0, rV = 0.0, kd = 0.0;
    UnitGeo f{};
    St5 own{1.0, 1.0, 0.0, 0.0, 1.0}, bnd{};
    int nbc = -1, ft = -1;
    bool scaled = false, swap = false;
    if (act) {
        ry = 1.0 / b0.cy[c];
        rV = 1.0 / b0.vs[c];
        own = load_state(b0.cur, c);
        const int g = d.gstart[c] + j;
        if (g < d.gstart[c + 1]) {
            const int su = d.s_unit[g], u = su >> 1;
            const bool twin = su & 1;
            const size_t nu = d.n_units;
            const double* r = b0.ugeo + u;
            ft = d.sinfo[g] & SI_TYPE_MASK;
            nbc = twin ? d.u_cell[u] : d.u_nb[u];
            f.flags = reinterpret_cast<const uint32_t*>(b0.ugeo + kUnitGeoRows * nu)[u];
            f.n1 = r[0];
            f.n2 = r[nu];
            f.S = r[2 * nu];
            kd = mul_rn(P.kurant, r[(twin ? 4 : 3) * nu]);
            f.kroO = r[5 * nu];
            f.kpO = r[6 * nu];
            f.CO = r[7 * nu];
            f.SO = r[8 * nu];
            f.kroN = r[9 * nu];
            f.kpN = r[10 * nu];
            f.CN = r[11 * nu];
            f.SN = r[12 * nu];
            scaled = f.flags & (twin ? 2u : 1u);
            // the twin evaluates the face as the main face's owner does,
            // unless the radial scaling switches between the two cells
            const bool same = f.flags == 0u || f.flags == 3u;
            swap = twin && same;
            if (twin && !same) {
                f.n1 = -f.n1;
                f.n2 = -f.n2;
            }
            if (ft == G_USUALY) {
                if (twin) {  // own side first
                    double w = f.kroO; f.kroO = f.kroN; f.kroN = w;
                    w = f.kpO; f.kpO = f.kpN; f.kpN = w;
                    w = f.CO; f.CO = f.CN; f.CN = w;
                    w = f.SO; f.SO = f.SN; f.SN = w;
                }
            } else {
                St5 L;
                plain_boundary(P, ft, own, scaled, f, L, bnd);  // the constant state of Inner_sphere / Input
                f.kroN = bnd.ro;
                f.kpN = bnd.p;
                f.CN = bnd.u;
                f.SN = bnd.v;
                f.distn = bnd.Q;
            }
        }
    }
    const double sg = swap ? -f.S : f.S;
    double dt = *b0.dt_cur, dt_prev = dt;
    int nro = 0, npc = 0;
    for (int st = 0; st < nsteps; st++) {
        const StepBuffers& b = (st & 1) ? b1 : b0;
        double F[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        double t = act ? 10000000.0 : inf;  // `time` of Setka.cpp:5222
        if (ft >= 0) {
            St5 L = own, R;
            if (ft == G_USUALY) {
                R.ro = __ldcg(b.cur[0] + nbc);
                R.p = __ldcg(b.cur[1] + nbc);
                R.u = __ldcg(b.cur[2] + nbc);
                R.v = __ldcg(b.cur[3] + nbc);
                R.Q = __ldcg(b.cur[4] + nbc);
                if (scaled) {
                    L = plain_scale(L, f.kroO, f.kpO, f.CO, f.SO);
                    R = plain_scale(R, f.kroN, f.kpN, f.CN, f.SN);
                }
                if (swap) {
                    const St5 w = L;
                    L = R;
                    R = w;
                }
            } else if (ft == G_INNER_SPHERE || ft == G_INPUT) {
                if (ft == G_INNER_SPHERE) {
                    L.ro = mul_rn(L.ro, f.kroO);
                    L.p = mul_rn(L.p, f.kpO);
                }
                R = St5{f.kroN, f.kpN, f.CN, f.SN, f.distn};
            } else {
                plain_boundary(P, ft, own, scaled, f, L, R);
            }
            const double UU = plain_flux<TF>(P, L, R, f.n1, f.n2, F);
#pragma unroll
            for (int k = 0; k < 5; k++) F[k] = mul_rn(F[k], sg);
            t = dmin_ref(t, dt_candidate(kd / UU));
        }
        // the cell's slots in Grans order (a face that is not there adds 0)
        double Pt[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int k = 0; k < 5; k++) Pt[k] = Pt[k] + __shfl_sync(full, F[k], q0 + i);
        if (act) {
            int ro1 = 0, p1 = 0;
            own = plain_update(P, own, Pt, dt, rV, ry, ro1, p1);
            if (j == 0) {
                nro += ro1;
                npc += p1;
                b.nxt[0][c] = own.ro;
                b.nxt[4][c] = own.Q;
            } else {
                b.nxt[j][c] = j == 1 ? own.p : j == 2 ? own.u : own.v;
            }
        }
        unsigned long long* acc = plain_acc(b0.dt_acc, st);
        t = block_min_nonneg(t, sm);
        if (threadIdx.x == 0 && t < inf) atomicMin(acc, static_cast<unsigned long long>(__double_as_longlong(t)));
        grid.sync();
        dt_prev = dt;
        dt = plain_dt(__ldcg(acc));
        if (tid == 0) *plain_acc(b0.dt_acc, st + 2) = 0x7ff0000000000000ULL;
    }
    if (nro) atomicAdd(&b0.counters[0], static_cast<unsigned long long>(nro));
    if (npc) atomicAdd(&b0.counters[1], static_cast<unsigned long long>(npc));
    if (tid == 0) {
        const StepBuffers& b = ((nsteps - 1) & 1) ? b1 : b0;
        *b.dt_next = dt;
        *const_cast<double*>(b.dt_cur) = dt_prev;
    }
}

// `nsteps` Go_stationary steps of many instances in one launch.  The
// instances share the mesh (topology and geometry) and have their own
// parameters (inflow and inner-wind states), state buffers, flux slots and
// dt words, and never exchange data: one thread-block cluster advances one
// instance, the phases of a step separated by cluster barriers, and the CFL
// minimum goes from block to block through distributed shared memory (no
// atomics, no dt words inside the call).  A block owns a contiguous chunk of
// the instance's units and cells; the cluster is the largest at which every
// instance is resident (launch_stationary_batch).  `active` lists the
// instances advanced by this launch (the others keep their state).
// Bound by the latency of the unit and cell bodies at 16 warps per SM.  With
// one grid of blocks for all instances and three grid barriers per step, 32
// instances of 90 x 60 cells took 72.8 us per step, here 33; 60: 167 and 69;
// 16 of 60 x 40 cells: 35.5 and 17.5; one of 90 x 60: 14.9 and 14.6.  256
// threads at 128 registers: 512 x 1 block per SM measured 2% slower, 256
// threads at 80 or 64 registers 26-40% (spills), 384 at 80 15%.
constexpr int kClusterThreads = 256, kClusterMax = 16;
template <typename TF>
__global__ void __launch_bounds__(kClusterThreads, 2)
    stationary_cluster_kernel(DevMesh d, const PlainInstance* __restrict__ inst, const int* __restrict__ active,
                              int nsteps) {
    __shared__ PlainInstance I;
    __shared__ double sm[32];
    __shared__ double mins[kClusterMax];  // the CFL minimum of every block of the cluster, written by that block
    cg::cluster_group cl = cg::this_cluster();
    const int nb = static_cast<int>(cl.num_blocks()), rank = static_cast<int>(cl.block_rank());
    {
        static_assert(sizeof(PlainInstance) % 8 == 0, "copied as 8-byte words");
        const unsigned long long* s8 = reinterpret_cast<const unsigned long long*>(inst + active[blockIdx.x / nb]);
        unsigned long long* d8 = reinterpret_cast<unsigned long long*>(&I);
        for (int i = threadIdx.x; i < static_cast<int>(sizeof(PlainInstance) / 8); i += blockDim.x) d8[i] = s8[i];
    }
    cl.sync();  // the descriptor is in; every block of the cluster runs before one writes into another's memory
    auto cut = [&](int n, int r) { return static_cast<int>(static_cast<long long>(n) * r / nb); };
    const int u0 = cut(d.n_units, rank), u1 = cut(d.n_units, rank + 1);
    const int c0 = cut(d.n_cells, rank), c1 = cut(d.n_cells, rank + 1);
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    bool any = false;
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) any |= !(d.cflags[c] & CF_CENTR);
    double dt = *I.b[0].dt_cur, dt_prev = dt, tmark = inf;
    int nro = 0, npc = 0;
    for (int st = 0; st < nsteps; st++) {
        const StepBuffers& b = I.b[st & 1];
        double t = any ? 10000000.0 : inf;  // `time` of Setka.cpp:5222
        for (int u = u0 + threadIdx.x; u < u1; u += blockDim.x)
            t = dmin_ref(t, dt_candidate(stationary_unit_body<TF>(d, I.P, b, I.fl, u)));
        t = block_min_nonneg(t, sm);
        if (threadIdx.x < nb) *cl.map_shared_rank(&mins[rank], threadIdx.x) = t;
        cl.sync();
        double m = mins[0];
        for (int k = 1; k < nb; k++) m = dmin_ref(m, mins[k]);
        for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x)
            stationary_update_body(d, I.P, b, I.fl, c, dt, tmark, nro, npc);
        dt_prev = dt;
        dt = (m == inf) ? 100000000.0 : m;
        cl.sync();
    }
    if (nro) atomicAdd(&I.b[0].counters[0], static_cast<unsigned long long>(nro));
    if (npc) atomicAdd(&I.b[0].counters[1], static_cast<unsigned long long>(npc));
    if (rank == 0 && threadIdx.x == 0) {
        const StepBuffers& b = I.b[(nsteps - 1) & 1];
        *b.dt_next = dt;
        *const_cast<double*>(b.dt_cur) = dt_prev;
    }
}

// Go_5_komponent__MK2 face reconstruction of one side (Setka.cpp:10213-10276)
// for a Usualy face: owner M (state Ms, centre Mx,My, flags mf), across the
// face the cell So; Sd = Sosed_down of the face as seen from M.
__device__ __forceinline__ St5 mk2_usualy_side(const double* const* st, const double* cx, const double* cy,
                                               const double* rp, double fx, double fy, double dis, double pdis,
                                               const St5& Ms, double Mx, double My, double rpM, uint32_t mf, int So,
                                               int Sd, bool tracked, int* status) {
    if (mf & CF_C1) {
        const double radius = sqrt(sq(Mx) + sq(My));
        St5 o = Ms;
        o.ro = o.ro * sq(radius) / sq(dis);
        o.Q = o.Q * sq(radius) / sq(dis);
        o.p = o.p * (rpM / pdis);
        polar_perenos(Mx, My, fx, fy, o.u, o.v);
        tvd_radial(st, cx, cy, rp, fx, fy, Ms, Mx, My, rpM, So, Sd, (mf & CF_AXIS) != 0, pdis, o.ro, o.p);
        return o;
    }
    return tvd_usualy(st, cx, cy, fx, fy, Ms, Mx, My, So, Sd, (mf & CF_AXIS) != 0, tracked, status);
}
// The same for a face unit that has computed the distances already: rM, rS
// = |centroid| of M and So, dM, dS = face centre to those centroids.
__device__ __forceinline__ St5 mk2_usualy_side_d(const double* const* st, const double* cx, const double* cy,
                                                 const double* rp, double fx, double fy, double dis, double pdis,
                                                 const St5& Ms, double Mx, double My, double rpM, uint32_t mf, int So,
                                                 int Sd, bool tracked, double rM, double rS, double dM, double dS,
                                                 int* status) {
    if (mf & CF_C1) {
        const double radius = rM;
        St5 o = Ms;
        o.ro = o.ro * sq(radius) / sq(dis);
        o.Q = o.Q * sq(radius) / sq(dis);
        o.p = o.p * (rpM / pdis);
        polar_perenos(Mx, My, fx, fy, o.u, o.v);
        tvd_radial_d(st, cx, cy, rp, fx, fy, Ms, Mx, My, rpM, So, Sd, (mf & CF_AXIS) != 0, pdis, dis, rM, rS, dM, dS,
                     o.ro, o.p);
        return o;
    }
    return tvd_usualy_d(st, cx, cy, fx, fy, Ms, Mx, My, So, Sd, (mf & CF_AXIS) != 0, tracked, dM, dS, status);
}

// One MK2 face unit before the grid moves (Setka.cpp:10204-10276): the two
// reconstructed face states (TVD / radial TVD / boundary states), the face
// normal, S = |AB| (yA + yB) / 2, the face centre and the two CFL distances
// (negative: that side is not updated this step).  Everything here reads the
// points before the motion (X, Y) and the cached centroids, never the moved
// points, so it may run before or after the rails.
struct RecUnit {
    St5 a, o;                  // owner side, other side
    double n1, n2, S, x2, y2;  // face normal, S, face centre
    double dist, distn;        // owner / other centroid to the face centre, -1 if not updated
};

// L1 prefetch of one global address (no register, no wait).
__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// Prefetch into L1 of everything mk2_recon_unit / mk2_flux_unit gather for
// face unit u: state rows and centroids of the owner, the neighbour and both
// Sosed_down cells (and |c|^(2 gamma) where RP: the radial reconstruction),
// the end points before and after the motion.
template <bool RP>
__device__ __forceinline__ void mk2_prefetch_unit(const DevMesh& d, const StepBuffers& b, int u) {
    const int K = d.u_cell[u], nb = d.u_nb[u], A = d.u_A[u], B = d.u_B[u];
    const int sd = d.u_sd[u], sd2 = d.u_sd2[u];
    auto cell = [&](int c) {
#pragma unroll
        for (int k = 0; k < 5; k++) prefetch_l1(b.cur[k] + c);
        prefetch_l1(b.cx + c);
        prefetch_l1(b.cy + c);
        if (RP) prefetch_l1(b.rp + c);
    };
    cell(K);
    if (nb >= 0) cell(nb);
    if (sd >= 0) cell(sd);
    if (sd2 >= 0) cell(sd2);
    prefetch_l1(d.X + A);
    prefetch_l1(d.Y + A);
    prefetch_l1(d.X + B);
    prefetch_l1(d.Y + B);
    prefetch_l1(d.X2 + A);
    prefetch_l1(d.Y2 + A);
    prefetch_l1(d.X2 + B);
    prefetch_l1(d.Y2 + B);
}

// GROUP: the unit group the caller knows the unit to be in, so that branches
// drop out at compile time: kPlainGroup [0, u_c1) (a Usualy face, neither
// cell C_1, not tracked), kC1Group [u_c1, u_tr0) (a Usualy face with a C_1
// side, not tracked), kAnyGroup (no assumption).
constexpr int kPlainGroup = 0, kC1Group = 1, kAnyGroup = 2;
template <int GROUP = kAnyGroup>
__device__ __forceinline__ void mk2_recon_unit(const DevMesh& d, const gelios_params& P, const StepBuffers& b, int u,
                                               RecUnit& r, int* status) {
    constexpr bool PLAIN = GROUP == kPlainGroup, USUALY = GROUP != kAnyGroup;
    const int K = d.u_cell[u], nb = d.u_nb[u];
    const uint32_t info = d.u_info[u];
    const double x = b.cx[K], y = b.cy[K];
    // centroid radii (where a radial reconstruction needs them) and
    // face-centre-to-centroid distances, computed once for the R11 test, the
    // CFL candidates and both reconstructions
    const double aK = sq(x) + sq(y);
    const bool procK = !(aK < d.r11_sq);
    const double rK = PLAIN ? 0.0 : sqrt(aK);
    double x3 = 0.0, y3 = 0.0, rN = 0.0;
    bool procN = false;
    if (nb >= 0) {
        x3 = b.cx[nb];
        y3 = b.cy[nb];
        const double aN = sq(x3) + sq(y3);
        procN = !(aN < d.r11_sq);
        rN = PLAIN ? 0.0 : sqrt(aN);
    }
    const int A = d.u_A[u], B = d.u_B[u];
    const double xa = d.X[A], ya = d.Y[A], xb = d.X[B], yb = d.Y[B];
    const double x2 = (xa + xb) / 2.0, y2 = (ya + yb) / 2.0;
    const double dK = sqrt(sq(x - x2) + sq(y - y2));
    const double dN = sqrt(sq(x3 - x2) + sq(y3 - y2));
    {
        double t1 = xb - xa, t2 = yb - ya;
        const double nn = sqrt(sq(t1) + sq(t2));
        t1 = t1 / nn;
        t2 = t2 / nn;
        r.n1 = t2;
        r.n2 = -t1;
        r.S = sqrt(sq(xb - xa) + sq(yb - ya)) * (ya + yb) * 0.5;
        r.x2 = x2;
        r.y2 = y2;
        r.dist = procK ? dK : -1.0;
        r.distn = procN ? dN : -1.0;
    }
    if (!(procK || procN)) return;
    const int ft = USUALY ? static_cast<int>(G_USUALY) : static_cast<int>(info & SI_TYPE_MASK);
    const uint32_t cf = (info >> UI_CF_OWN) & (PLAIN ? (15u & ~CF_C1) : 15u);
    const double g2 = 2 * P.gamma;
    const St5 par1 = load_state(b.cur, K);
    St5 par11 = par1;
    St5 par2 = get_par(P, ft, par1, b.cur, nb, x2, y2);
    const double dis = sqrt(sq(x2) + sq(y2));
    const bool tracked = !USUALY && (info & SI_GOD) != 0;
    const uint32_t nbf = (info >> UI_CF_NB) & (PLAIN ? (15u & ~CF_C1) : 15u);
    const bool radial = ((cf & CF_C1) && (ft == G_USUALY || ft == G_AXIS)) || ft == G_INNER_SPHERE ||
                        (ft == G_USUALY && (nbf & CF_C1));
    const double pdis = radial ? pow2g(dis, g2) : 1.0;
    if (ft == G_USUALY) {
        r.a = mk2_usualy_side_d(b.cur, b.cx, b.cy, b.rp, x2, y2, dis, pdis, par1, x, y, b.rp[K], cf, nb, d.u_sd[u],
                                tracked, rK, rN, dK, dN, status);
        r.o = mk2_usualy_side_d(b.cur, b.cx, b.cy, b.rp, x2, y2, dis, pdis, par2, x3, y3, b.rp[nb], nbf, K,
                                d.u_sd2[u], tracked, rN, rK, dN, dK, status);
        return;
    }
    if (ft == G_INNER_SPHERE) {
        const double radius = rK;
        par11.ro = par11.ro * sq(radius) / sq(dis);
        par11.Q = par11.Q * sq(radius) / sq(dis);
        par11.p = par11.p * (b.rp[K] / pdis);
    } else if (ft == G_AXIS) {
        if (cf & CF_C1) {
            const double radius = rK;
            par11.ro = par11.ro * sq(radius) / sq(dis);
            par11.Q = par11.Q * sq(radius) / sq(dis);
            par11.p = par11.p * (b.rp[K] / pdis);
            polar_perenos(x, y, x2, y2, par11.u, par11.v);
        } else {
            par11 = tvd_axis(b.cur, b.cx, b.cy, x2, y2, par1, x, y, d.u_sd[u]);
        }
        par2 = par11;
        par2.v = -par2.v;
    }
    r.a = par11;
    r.o = par2;
}

// The flux of one MK2 face unit once the grid has moved (Setka.cpp:10198-10209,
// 10335-10393): face speed W from the moved points, HLL (`metod 0`), exact
// Godunov sampled at W on tracked faces (star pressure pstar solved before the
// motion), F.S into the unit's flux rows, CFL candidates.
template <typename TF, bool TRACKED>
__device__ __forceinline__ void mk2_flux_unit(const DevMesh& d, const gelios_params& P, const StepBuffers& b, int u,
                                              const RecUnit& r, double* __restrict__ fl, const double* pstar,
                                              double& tmin_u, int* status) {
    const bool procK = !(r.dist < 0.0), procN = !(r.distn < 0.0);
    if (!(procK || procN)) return;
    const size_t nu = d.n_units;
    const double dt = *b.dt_cur;
    const int A = d.u_A[u], B = d.u_B[u];
    const double x4 = (d.X2[A] + d.X2[B]) / 2.0, y4 = (d.Y2[A] + d.Y2[B]) / 2.0;
    const double W = ((x4 - r.x2) * r.n1 + (y4 - r.y2) * r.n2) / dt;
    const bool np = (d.u_info[u] & SI_NP) != 0;
    FluxOut<double> F;
    double UU;
    if constexpr (sizeof(TF) == 8) UU = hll_lean(P.gamma, r.a, r.o, W, r.n1, r.n2, F);
    else UU = hllc_flux<TF>(P.gamma, P.kurant, r.a, r.o, W, r.n1, r.n2, 1.0, 0, np, F);
    const double S = r.S;
    double fm0 = F.P0 * S, fm1 = F.P1 * S, fm2 = F.P2 * S, fm3 = F.P3 * S;
    double UG = 1.0;
    if (TRACKED) {
        double q1[5] = {r.a.ro, r.a.p, r.a.u, r.a.v, 0.0};
        double q2[5] = {r.o.ro, r.o.p, r.o.u, r.o.v, 0.0};
        double nv[3] = {r.n1, r.n2, 0.0};
        double qq[5], ds[3];
        UG = godunov_dev<false>(P.gamma, P.kurant, q1, q2, nv, qq, ds, W, 1.0, P.godunov_max_iter, status, pstar);
        fm0 = qq[0] * S;
        fm1 = qq[1] * S;
        fm2 = qq[2] * S;
        fm3 = qq[4] * S;
    }
    const double fq = F.PQ * S;
    fl[0 * nu + u] = fm0;
    fl[1 * nu + u] = fm1;
    fl[2 * nu + u] = fm2;
    fl[3 * nu + u] = fm3;
    fl[4 * nu + u] = fq;
    // the CFL candidates kurant * distance / speed of the updated sides and of
    // both solvers (Setka.cpp:10359, 10366): the least is that of the smaller
    // distance and the larger speed (a NaN speed gives none)
    const double dm = procK ? (procN ? dmin_ref(r.dist, r.distn) : r.dist) : r.distn;
    const double us = TRACKED && UG > UU ? UG : UU;
    tmin_u = dmin_ref(tmin_u, P.kurant * dm / us);
    if (TRACKED && !(us == us)) tmin_u = dmin_ref(tmin_u, P.kurant * dm / UG);
}

// Rows of the tracked units' reconstruction (kRecRows rows of n_tracked
// doubles; row r of tracked unit i at rec[r * n_tracked + i]).
__device__ __forceinline__ void rec_store(double* __restrict__ rec, size_t n, int i, const RecUnit& r) {
    const double v[kRecRows] = {r.a.ro, r.a.p, r.a.u, r.a.v, r.a.Q, r.o.ro, r.o.p, r.o.u, r.o.v,
                                r.o.Q, r.n1,  r.n2,  r.S,   r.x2,  r.y2,  r.dist, r.distn};
#pragma unroll
    for (int k = 0; k < kRecRows; k++) rec[k * n + i] = v[k];
}
__device__ __forceinline__ RecUnit rec_load(const double* __restrict__ rec, size_t n, int i) {
    RecUnit r;
    r.a.ro = rec[0 * n + i];
    r.a.p = rec[1 * n + i];
    r.a.u = rec[2 * n + i];
    r.a.v = rec[3 * n + i];
    r.a.Q = rec[4 * n + i];
    r.o.ro = rec[5 * n + i];
    r.o.p = rec[6 * n + i];
    r.o.u = rec[7 * n + i];
    r.o.v = rec[8 * n + i];
    r.o.Q = rec[9 * n + i];
    r.n1 = rec[10 * n + i];
    r.n2 = rec[11 * n + i];
    r.S = rec[12 * n + i];
    r.x2 = rec[13 * n + i];
    r.y2 = rec[14 * n + i];
    r.dist = rec[15 * n + i];
    r.distn = rec[16 * n + i];
    return r;
}

// The tracked face units (grouped in [u_tr0, u_tr1)) are reconstructed before
// the motion: their exact Riemann problems are solved while the grid moves.
__global__ void __launch_bounds__(128) mk2_recon_tracked_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                                double* __restrict__ rec) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nt = d.u_tr1 - d.u_tr0;
    int status = 0;
    if (i < nt) {
        RecUnit r;
        r.a = St5{};
        r.o = St5{};
        mk2_recon_unit(d, P, b, d.u_tr0 + i, r, &status);
        rec_store(rec, nt, i, r);
    }
    if (status) atomicOr(b.status, status);
}

// Tracked units after the motion: sampling of the solved Riemann problems
// at the face speed (one thread per unit).
template <typename TF>
__global__ void __launch_bounds__(32) mk2_flux_tracked_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                              const double* __restrict__ rec, double* __restrict__ fl,
                                                              const double* __restrict__ pstar) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nt = d.u_tr1 - d.u_tr0;
    double tmin_u = __longlong_as_double(0x7ff0000000000000LL);
    int status = 0;
    if (i < nt) {
        const RecUnit r = rec_load(rec, nt, i);
        mk2_flux_unit<TF, true>(d, P, b, d.u_tr0 + i, r, fl, pstar + i, tmin_u, &status);
    }
    block_reduce_commit(tmin_u, 0, 0, status, b.dt_acc, b.counters, b.status);
}

// The plain interior face units [0, u_c1) after the motion, reconstruction and
// flux in one pass: the reconstructed states stay in registers (no per-unit
// scratch); F.S once per unit, as its owner sees it.  Compiled without the
// branches that the C_1 and the one-sided units take (mk2_face_rest_kernel).
// PF: every gathered address of the unit is prefetched into L1 as soon as
// the unit's indices are in (mk2_prefetch_unit), so that the loads of the
// reconstruction's later levels hit L1 instead of waiting for L2 / DRAM one
// level at a time; the arithmetic is the same code.
template <typename TF, int MINB, bool PF>
__global__ void __launch_bounds__(128, MINB) mk2_face_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                           double* __restrict__ fl, int n_launch) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    double tmin_u = __longlong_as_double(0x7ff0000000000000LL);
    int status = 0;
    if (u < n_launch) {
        if (PF) mk2_prefetch_unit<false>(d, b, u);
        RecUnit r;
        r.a = St5{};
        r.o = St5{};
        mk2_recon_unit<kPlainGroup>(d, P, b, u, r, &status);
        mk2_flux_unit<TF, false>(d, P, b, u, r, fl, nullptr, tmin_u, &status);
    }
    block_reduce_commit(tmin_u, 0, 0, status, b.dt_acc, b.counters, b.status);
}

// The C_1 interior and the one-sided units in one launch (each block one
// kind), so that a small grid has one kernel less in its chain; 38 us on the
// 938k grid (41 + 12 in two launches with the flux of hllc_flux; ncu).
template <typename TF, int MINB, bool PF>
__global__ void __launch_bounds__(128, MINB) mk2_face_rest_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                                  double* __restrict__ fl, int n_one_blocks) {
    double tmin_u = __longlong_as_double(0x7ff0000000000000LL);
    int status = 0;
    RecUnit r;
    r.a = St5{};
    r.o = St5{};
    if (static_cast<int>(blockIdx.x) < n_one_blocks) {
        const int u = d.u_tr1 + blockIdx.x * blockDim.x + threadIdx.x;
        if (u < d.n_units) {
            mk2_recon_unit<kAnyGroup>(d, P, b, u, r, &status);
            mk2_flux_unit<TF, false>(d, P, b, u, r, fl, nullptr, tmin_u, &status);
        }
    } else {
        const int u = d.u_c1 + (blockIdx.x - n_one_blocks) * blockDim.x + threadIdx.x;
        if (u < d.u_tr0) {
            if (PF) mk2_prefetch_unit<true>(d, b, u);
            mk2_recon_unit<kC1Group>(d, P, b, u, r, &status);
            mk2_flux_unit<TF, false>(d, P, b, u, r, fl, nullptr, tmin_u, &status);
        }
    }
    block_reduce_commit(tmin_u, 0, 0, status, b.dt_acc, b.counters, b.status);
}

// Star pressure of the exact Godunov problem of every tracked-face unit
// (Solvers.cpp:1174-1305).  It depends on the reconstructed states and on
// the face normal before the motion, not on the face speed, so it runs on a
// side stream while the grid moves; mk2_flux_tracked_kernel samples the
// solution at the face speed afterwards.  One warp per unit (warp-cooperative
// bisection); pstar[i] belongs to unit u_tr0 + i.
__global__ void __launch_bounds__(64) mk2_tracked_solve_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                               const double* __restrict__ rec,
                                                               double* __restrict__ pstar) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nt = d.u_tr1 - d.u_tr0;
    if (i >= nt) return;
    int status = 0;
    const size_t n = nt;
    // a unit with neither side updated has no flux (rows 15 and 16)
    if (rec[15 * n + i] < 0.0 && rec[16 * n + i] < 0.0) return;
    double q1[5] = {rec[0 * n + i], rec[1 * n + i], rec[2 * n + i], rec[3 * n + i], 0.0};
    double q2[5] = {rec[5 * n + i], rec[6 * n + i], rec[7 * n + i], rec[8 * n + i], 0.0};
    double nv[3] = {rec[10 * n + i], rec[11 * n + i], 0.0};
    double qq[5], ds[3], p = 0.0;
    godunov_dev<true>(P.gamma, P.kurant, q1, q2, nv, qq, ds, 0.0, 1.0, P.godunov_max_iter, &status, nullptr, &p);
    if ((threadIdx.x & 31) == 0) {
        pstar[i] = p;
        if (status) atomicOr(b.status, status);
    }
}

// The term of the MK2 cell update that depends neither on the fluxes nor on
// the motion: the charge-exchange source Get_Sourse_MK1 (Cell.cpp:498-665).
// Runs on a side stream while surface tracking and the rails move the grid.
// aux rows: q1, q2, q3
// 32 cells per warp in two phases, every lane busy in both.  Cell phase: one
// lane per cell decides whether the cell takes part, finds the bracket of
// the radial interpolation, loads the cell's state and interpolates the
// k_u, k_v, k_T factors; the per-cell values go to shared memory.  Species
// phase: four rounds of eight cells x four hydrogen species, one (cell,
// species) pair per lane: the species' moments at the cell and its exchange
// rates; the four rates are summed on the cell's first species lane in the
// reference's order (H1 + H2 + H3 + H4), which writes the cell's q1..q3.
__global__ void __launch_bounds__(128, GELIOS_SOURCE_MINB) mk2_source_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                                             double* __restrict__ aux) {
    // per-cell values of the block's 128 cells, one row per quantity
    __shared__ double sd[10][128];  // u, v, ro, p/ro, u^2+v^2, 1/(r1-r2), rr-r2, k_u, k_v, k_T
    __shared__ int si[3][128];      // K_do, K_posle, flags (1 takes part, 2 bracket found, 4 interpolated)
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wbase = threadIdx.x & ~31;
    const int c0 = blockIdx.x * blockDim.x + wbase;  // the warp's first cell
    int status = 0;
    {
        const int c = c0 + lane, t = threadIdx.x;
        int flags = 0, K_do = -1, K_posle = -1;
        double e[10] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (c < d.n_cells) {
            const double x = b.cx[c], y = b.cy[c];
            const double rr = sqrt(sq(x) + sq(y));
            const bool proc = !(rr < P.R11);
            const bool interp = proc && rr > P.src_rmin && rr < P.src_rmax && x >= 0.0;
            bool ok = true;
            if (interp) {
                int2 cached;
                ok = source_bracket(d, c, rr, K_do, K_posle, &status, &cached);
                if (ok && d.src_lo_out && cached.x != K_do) d.src_lo_out[c] = make_int2(K_do, K_posle);
            }
            if (proc && ok) {
                const St5 par1 = load_state(b.cur, c);
                e[0] = par1.u;
                e[1] = par1.v;
                e[2] = par1.ro;
                e[3] = par1.p / par1.ro;
                e[4] = sq(par1.u) + sq(par1.v);
                if (interp) {
                    const double r1 = d.r_istoch[K_do], r2 = d.r_istoch[K_posle];
                    const double ir = 1.0 / (r1 - r2), dr = rr - r2;
                    auto lin = [&](double t1, double t2) { return (t1 - t2) * ir * dr + t2; };
                    e[5] = ir;
                    e[6] = dr;
                    e[7] = lin(d.ku[K_do], d.ku[K_posle]);
                    e[8] = lin(d.kv[K_do], d.kv[K_posle]);
                    e[9] = lin(d.kT[K_do], d.kT[K_posle]);
                } else {
                    e[7] = d.ku[c];
                    e[8] = d.kv[c];
                    e[9] = d.kT[c];
                }
            }
            flags = (proc ? 1 : 0) | (ok ? 2 : 0) | (interp ? 4 : 0);
        }
#pragma unroll
        for (int k = 0; k < 10; k++) sd[k][t] = e[k];
        si[0][t] = K_do;
        si[1][t] = K_posle;
        si[2][t] = flags;
    }
    __syncwarp();
    const int sp = lane & 3, q0 = lane & ~3;
#pragma unroll 1
    for (int r = 0; r < 4; r++) {
        const int t = wbase + 8 * r + (lane >> 2);  // the lane's cell, as a block slot
        const int c = c0 + 8 * r + (lane >> 2);
        const int flags = c < d.n_cells ? si[2][t] : 0;
        double nuu = 0.0, nuv = 0.0, nue = 0.0;
        if ((flags & 3) == 3) {
            double uH, vH, roH, TH;
            if (flags & 4) {
                const int K_do = si[0][t], K_posle = si[1][t];
                const double ir = sd[5][t], dr = sd[6][t];
                auto lin = [&](double t1, double t2) { return (t1 - t2) * ir * dr + t2; };
                uH = lin(d.Hu[4 * K_do + sp], d.Hu[4 * K_posle + sp]);
                vH = lin(d.Hv[4 * K_do + sp], d.Hv[4 * K_posle + sp]);
                roH = lin(d.Hn[4 * K_do + sp], d.Hn[4 * K_posle + sp]);
                TH = lin(d.HT[4 * K_do + sp], d.HT[4 * K_posle + sp]);
            } else {
                uH = d.Hu[4 * c + sp];
                vH = d.Hv[4 * c + sp];
                roH = d.Hn[4 * c + sp];
                TH = d.HT[4 * c + sp];
            }
            // th = 2 pH / roH with pH = TH roH / 2, or pH = 0 where there is no hydrogen (Cell.cpp:590-594)
            if (roH <= 0.0) {
                roH = 0.0000001;
                TH = 0.0;
            }
            source_rates_th(P, uH, vH, roH, TH, sd[0][t], sd[1][t], sd[2][t], sd[3][t], sd[4][t], nuu, nuv, nue);
        }
        double su[3], sv[3], se[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            su[j] = __shfl_sync(full, nuu, q0 + 1 + j);
            sv[j] = __shfl_sync(full, nuv, q0 + 1 + j);
            se[j] = __shfl_sync(full, nue, q0 + 1 + j);
        }
        if (sp == 0 && (flags & 1)) {
            const size_t n = d.n_cells;
            double q1 = 0.0, q2 = 0.0, q3 = 0.0;
            if (flags & 2) {
                const double Mu = P.src_coef * (nuu + su[0] + su[1] + su[2]);
                const double Mv = P.src_coef * (nuv + sv[0] + sv[1] + sv[2]);
                const double MT = P.src_coef * (nue + se[0] + se[1] + se[2]);
                q1 = Mu * sd[7][t];
                q2 = Mv * sd[8][t];
                q3 = MT * sd[9][t];
            }
            aux[0 * n + c] = q1;
            aux[1 * n + c] = q2;
            aux[2 * n + c] = q3;
        }
    }
    if (status) atomicOr(b.status, status);
}

// Go_5_komponent__MK2 cell update (Setka.cpp:10386-10468) of cell c from its
// nf face slots' fluxes (fetch4 / fetch(k, j): row k of the cell's j-th slot,
// Grans order; fetch4 where there are four).  The area and rotated volume before the motion come from the cache
// (b.vs, b.vol); the cache is refilled for the next step from the moved
// points: centroid, and area and rotated volume of every cell but the C_centr
// ones (the points after the commit are these moved points, bit for bit),
// |centroid|^(2 gamma) of the cells flagged CF_RP.  For a quadrilateral
// Get_Volume and Get_Volume_posle are the same formula; other cells get the
// Get_Volume form for the cache.
template <typename Fetch4, typename Fetch>
__device__ __forceinline__ void mk2_update_cell(const DevMesh& d, const gelios_params& P, const StepBuffers& b, int c,
                                                int nf, Fetch4 fetch4, Fetch fetch, const double* __restrict__ aux,
                                                double& tmark, int& nro, int& npc) {
    const uint32_t cfl = d.cflags[c];
    const double x = b.cx[c], y = b.cy[c];
    double xn, yn, vs2 = 0.0, Volume2 = 0.0;
    // quadrilaterals: the corner indices in one 16-byte load (qcorner), so
    // the moved points are the second level of dependent loads, not the third
    const int4 qc = d.qcorner ? d.qcorner[c] : make_int4(-1, -1, -1, -1);
    if (qc.x >= 0) {
        // the four moved points once, in registers (the same operations as
        // centroid / area / volume_rotate)
        const double qx[4] = {d.X2[qc.x], d.X2[qc.y], d.X2[qc.z], d.X2[qc.w]};
        const double qy[4] = {d.Y2[qc.x], d.Y2[qc.y], d.Y2[qc.z], d.Y2[qc.w]};
        quad_geometry_lean(qx, qy, xn, yn, vs2, Volume2);
        if (!(cfl & CF_CENTR)) {
            b.vs_next[c] = vs2;
            b.vol_next[c] = Volume2;
        }
    } else if (const int n4 = d.cstart[c + 1] - d.cstart[c]; n4 == 4) {
        const int32_t* con = d.contour + d.cstart[c];
        const int p0 = con[0], p1 = con[1], p2 = con[2], p3 = con[3];
        const double qx[4] = {d.X2[p0], d.X2[p1], d.X2[p2], d.X2[p3]};
        const double qy[4] = {d.Y2[p0], d.Y2[p1], d.Y2[p2], d.Y2[p3]};
        quad_geometry_lean(qx, qy, xn, yn, vs2, Volume2);
        if (!(cfl & CF_CENTR)) {
            b.vs_next[c] = vs2;
            b.vol_next[c] = Volume2;
        }
    } else {
        const int s0 = d.cstart[c], n = d.cstart[c + 1] - s0;
        const int32_t* con = d.contour + s0;
        centroid(con, n, d.X2, d.Y2, xn, yn);
        if (!(cfl & CF_CENTR)) {
            vs2 = area(con, n, d.sA, d.sB, d.gstart[c], d.gstart[c + 1], d.X2, d.Y2, true);
            Volume2 = volume_rotate(con, n, d.X2, d.Y2);
            b.vs_next[c] = area(con, n, d.sA, d.sB, d.gstart[c], d.gstart[c + 1], d.X2, d.Y2, false);
            b.vol_next[c] = Volume2;
        }
    }
    b.cx_next[c] = xn;
    b.cy_next[c] = yn;
    if (cfl & CF_RP) b.rp_next[c] = pow2g(sqrt(sq(xn) + sq(yn)), 2 * P.gamma);
    if (sq(x) + sq(y) < d.r11_sq) return;
    tmark = dmin_ref(tmark, 10000000.0);  // `time` starts at 1e7 in every step (Setka.cpp:10141)
    const double dt = *b.dt_cur;
    double Pt0 = 0.0, Pt1 = 0.0, Pt2 = 0.0, Pt3 = 0.0, Pt4 = 0.0;
    if (nf == 4) {  // quadrilaterals: all slot loads in flight together
        double a[5][4];
#pragma unroll
        for (int k = 0; k < 5; k++)
#pragma unroll
            for (int j = 0; j < 4; j++) a[k][j] = fetch4(k, j);
        Pt0 = (((Pt0 + a[0][0]) + a[0][1]) + a[0][2]) + a[0][3];
        Pt1 = (((Pt1 + a[1][0]) + a[1][1]) + a[1][2]) + a[1][3];
        Pt2 = (((Pt2 + a[2][0]) + a[2][1]) + a[2][2]) + a[2][3];
        Pt3 = (((Pt3 + a[3][0]) + a[3][1]) + a[3][2]) + a[3][3];
        Pt4 = (((Pt4 + a[4][0]) + a[4][1]) + a[4][2]) + a[4][3];
    } else {
        for (int j = 0; j < nf; j++) {
            Pt0 = Pt0 + fetch(0, j);
            Pt1 = Pt1 + fetch(1, j);
            Pt2 = Pt2 + fetch(2, j);
            Pt3 = Pt3 + fetch(3, j);
            Pt4 = Pt4 + fetch(4, j);
        }
    }
    const St5 par1 = load_state(b.cur, c);
    const size_t nc = d.n_cells;
    const double q2_1 = aux[0 * nc + c], q2_2 = aux[1 * nc + c], q3 = aux[2 * nc + c];
    if (!(cfl & CF_CENTR)) {
        const double vs1 = b.vs[c];
        const double Volume = b.vol[c];
        const double ro = par1.ro, u = par1.u, v = par1.v, p = par1.p, Q = par1.Q;
        const double gm1 = P.gamma - 1, rg1 = 1.0 / gm1;
        const double rV2 = 1.0 / Volume2, VV = Volume * rV2;
        double ro3 = ro * VV - dt * (Pt0 * rV2);
        const double Q33 = Q * VV - (dt * rV2) * Pt4;
        if (ro3 <= 0.0) {
            ro3 = P.ro_floor;
            nro++;
        }
        const double rro3 = 1.0 / ro3;
        const double u3 = (ro * u * VV - dt * (Pt1 * rV2 - q2_1)) * rro3;
        const double v3 = (ro * v * VV - dt * ((Pt2 - p * 0.5 * (vs1 + vs2)) * rV2 - q2_2)) * rro3;
        double p3 =
            (((p * rg1 + ro * (u * u + v * v) * 0.5) * VV - dt * (Pt3 * rV2 - q3)) - 0.5 * ro3 * (u3 * u3 + v3 * v3)) *
            gm1;
        if (p3 <= 0) {
            p3 = P.p_floor;
            npc++;
        }
        b.nxt[0][c] = ro3;
        b.nxt[1][c] = p3;
        b.nxt[2][c] = u3;
        b.nxt[3][c] = v3;
        b.nxt[4][c] = Q33;
    } else {
        b.nxt[0][c] = par1.ro;
        b.nxt[1][c] = par1.p;
        b.nxt[2][c] = par1.u;
        b.nxt[3][c] = par1.v;
        b.nxt[4][c] = par1.Q;
    }
}

// The face units and the cell update of the moving-grid step, one tile of
// cells per block (tiles: spatially compact groups built at upload).  Phase
// 1: every face unit that touches the tile's cells, reconstruction and flux
// in registers, F.S (owner side) / -F.S (other side) into the tile-local
// slots in shared memory; a unit whose two cells lie in different tiles is
// evaluated by both (same inputs, same code: the same bits on both sides).
// Tracked units take the fluxes the tracked-face kernel left in `fl`.
// Phase 2: the update of every cell of the tile from its slots.  No flux
// leaves the SM.  The CFL candidate of a side is taken by the tile that holds
// that side's cell, so each is taken once.
template <typename TF, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) mk2_tile_kernel(DevMesh d, gelios_params P, StepBuffers b, TileView t,
                                                           const double* __restrict__ fl,
                                                           const double* __restrict__ aux) {
    extern __shared__ double sfl[];  // 5 rows of t.max_slots
    const int tile = blockIdx.x;
    const int ms = t.max_slots;
    const size_t nu = d.n_units;
    double tmin = __longlong_as_double(0x7ff0000000000000LL);
    int nro = 0, npc = 0, status = 0;
    const int f0 = t.fstart[tile], f1 = t.fstart[tile + 1];
    for (int j = f0 + threadIdx.x; j < f1; j += NT) {
        const int2 rec = t.faces[j];
        const int u = rec.x;
        const int own = rec.y & 0xffff, tw = (rec.y >> 16) & 0xffff;
        if (u >= d.u_tr0 && u < d.u_tr1) {
#pragma unroll
            for (int k = 0; k < 5; k++) {
                const double v = fl[k * nu + u];
                if (own != kTileNone) sfl[k * ms + own] = v;
                if (tw != kTileNone) sfl[k * ms + tw] = -v;
            }
            continue;
        }
        RecUnit r;
        r.a = St5{};
        r.o = St5{};
        mk2_recon_unit(d, P, b, u, r, &status);
        const bool procK = !(r.dist < 0.0), procN = !(r.distn < 0.0);
        if (!(procK || procN)) continue;
        const double dt = *b.dt_cur;
        const int A = d.u_A[u], B = d.u_B[u];
        const double x4 = (d.X2[A] + d.X2[B]) / 2.0, y4 = (d.Y2[A] + d.Y2[B]) / 2.0;
        const double W = ((x4 - r.x2) * r.n1 + (y4 - r.y2) * r.n2) / dt;
        const bool np = (d.u_info[u] & SI_NP) != 0;
        FluxOut<double> F;
        double UU;
        if constexpr (sizeof(TF) == 8) UU = hll_lean(P.gamma, r.a, r.o, W, r.n1, r.n2, F);
        else UU = hllc_flux<TF>(P.gamma, P.kurant, r.a, r.o, W, r.n1, r.n2, 1.0, 0, np, F);
        const double S = r.S;
        const double fm[5] = {F.P0 * S, F.P1 * S, F.P2 * S, F.P3 * S, F.PQ * S};
        if (own != kTileNone) {
#pragma unroll
            for (int k = 0; k < 5; k++) sfl[k * ms + own] = fm[k];
            if (procK) tmin = dmin_ref(tmin, P.kurant * r.dist / UU);
        }
        if (tw != kTileNone) {
#pragma unroll
            for (int k = 0; k < 5; k++) sfl[k * ms + tw] = -fm[k];
            if (procN) tmin = dmin_ref(tmin, P.kurant * r.distn / UU);
        }
    }
    __syncthreads();
    const int c0 = t.cstart[tile], c1 = t.cstart[tile + 1];
    for (int i = c0 + threadIdx.x; i < c1; i += NT) {
        const int c = t.cells[i];
        const int base = t.lbase[i];
        auto fetch = [&](int k, int jj) { return sfl[k * ms + base + jj]; };
        mk2_update_cell(d, P, b, c, d.gstart[c + 1] - d.gstart[c], fetch, fetch, aux, tmin, nro, npc);
    }
    block_reduce_commit(tmin, nro, npc, status, b.dt_acc, b.counters, b.status);
}

// The cell update alone, from the units' flux rows in global memory (the update
// phase of the tile kernel for the face-kernel arrangement).
// MODE kUpdAll: every cell, the 1e7 start of the CFL minimum folded into the
// accumulator (the reference's `time`, Setka.cpp:10141) when a cell takes
// part.  The pipelined step leaves that to its dt finalisation
// (in the surface kernel, commit with cap) and updates in two parts:
// kUpdEarly the listed cells (CF_EARLY), kUpdRest every other cell;
// kUpdAllNoMark every cell (its last step).
enum : int { kUpdAll = 0, kUpdEarly = 1, kUpdRest = 2, kUpdAllNoMark = 3 };
template <int MODE>
__global__ void __launch_bounds__(128, 8) mk2_update_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                          const double* __restrict__ fl,
                                                          const double* __restrict__ aux,
                                                          const int32_t* __restrict__ list, int n_list) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double tmark = __longlong_as_double(0x7ff0000000000000LL);
    int nro = 0, npc = 0;
    const size_t nu = d.n_units;
    int c = -1;
    if (MODE == kUpdEarly) {
        if (i < n_list) c = list[i];
    } else if (i < d.n_cells) {
        c = i;
        if (MODE == kUpdRest && (d.cflags[c] & CF_EARLY)) c = -1;
    }
    if (c >= 0) {
        const int g0 = d.gstart[c], nf = d.gstart[c + 1] - g0;
        int su[4] = {0, 0, 0, 0};
        if (nf == 4) {
#pragma unroll
            for (int j = 0; j < 4; j++) su[j] = d.s_unit[g0 + j];
        }
        mk2_update_cell(
            d, P, b, c, nf, [&](int k, int j) { return unit_flux(fl + k * nu, su[j]); },
            [&](int k, int j) { return unit_flux(fl + k * nu, d.s_unit[g0 + j]); }, aux, tmark, nro, npc);
    }
    if (MODE != kUpdAll) tmark = __longlong_as_double(0x7ff0000000000000LL);
    block_reduce_commit(tmark, nro, npc, 0, b.dt_acc, b.counters, b.status);
}

// Go_stationary_5_komponent_inner_MK2 cell update (Setka.cpp:7021-7210), one
// thread per cell: FP32 fluxes, and what inner_lanes_kernel does not take.
template <typename TF>
__global__ void __launch_bounds__(128) inner_cell_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                         const int32_t* __restrict__ list, int n_list) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double tmin_c = __longlong_as_double(0x7ff0000000000000LL);
    int nro = 0, npc = 0, status = 0;
    const double* const* st = b.cur;
    const int c = i < n_list ? list[i] : -1;
    if (c >= 0 && !(d.cflags[c] & CF_CENTR)) {
        const double dt = *b.dt_cur;
        const uint32_t cf = d.cflags[c];
        const int s0 = d.cstart[c], n = d.cstart[c + 1] - s0;
        const int32_t* con = d.contour + s0;
        const int g0 = d.gstart[c], g1 = d.gstart[c + 1];
        const St5 par1 = load_state(st, c);
        const double x = b.cx[c], y = b.cy[c];
        const double vs1 = area(con, n, d.sA, d.sB, g0, g1, d.X, d.Y, false);
        const double vs2 = area(con, n, d.sA, d.sB, g0, g1, d.X2, d.Y2, true);
        const double radius = sqrt(sq(x) + sq(y));
        const double Volume = volume_rotate(con, n, d.X, d.Y);
        const double g2 = 2.0 * P.gamma;
        double Pt0 = 0.0, Pt1 = 0.0, Pt2 = 0.0, Pt3 = 0.0, Pt4 = 0.0;
        double time = 10000000.0;
        for (int g = g0; g < g1; g++) {
            const int A = d.sA[g], B = d.sB[g];
            const uint32_t info = d.sinfo[g];
            const int ft = info & SI_TYPE_MASK;
            const double xa = d.X[A], ya = d.Y[A], xb = d.X[B], yb = d.Y[B];
            const double S = sqrt(sq(xb - xa) + sq(yb - ya)) * (ya + yb) * 0.5;
            const double x2 = (xa + xb) / 2.0, y2 = (ya + yb) / 2.0;
            const double dist = sqrt(sq(x - x2) + sq(y - y2));
            const int nb = d.snb[g];
            St5 par11 = par1;
            St5 par2 = get_par(P, ft, par1, st, nb, x2, y2);
            double t1 = xb - xa, t2 = yb - ya;
            const double nn = sqrt(sq(t1) + sq(t2));
            t1 = t1 / nn;
            t2 = t2 / nn;
            const double n1 = t2, n2 = -t1;
            int met = 1;
            const double dis = sqrt(sq(x2) + sq(y2));
            if (ft == G_USUALY) {
                const double x3 = b.cx[nb], y3 = b.cy[nb];
                const double dd = sqrt(sq(x3) + sq(y3));
                par11.ro = par11.ro * sq(radius) / sq(dis);
                par2.ro = par2.ro * sq(dd) / sq(dis);
                par11.Q = par11.Q * sq(radius) / sq(dis);
                par2.Q = par2.Q * sq(dd) / sq(dis);
                const double pdis = pow2g(dis, g2);
                par11.p = par11.p * (b.rp[c] / pdis);
                par2.p = par2.p * (b.rp[nb] / pdis);
                polar_perenos(x, y, x2, y2, par11.u, par11.v);
                polar_perenos(x3, y3, x2, y2, par2.u, par2.v);
                const uint32_t nbf = d.cflags[nb];
                if ((cf & CF_C1) && (nbf & CF_C1)) {
                    const St5 nbs = load_state(st, nb);
                    tvd_radial(st, b.cx, b.cy, b.rp, x2, y2, par1, x, y, b.rp[c], nb, d.ssd[g], (cf & CF_AXIS) != 0,
                               pdis, par11.ro, par11.p);
                    tvd_radial(st, b.cx, b.cy, b.rp, x2, y2, nbs, x3, y3, b.rp[nb], c, d.ssd2[g],
                               (nbf & CF_AXIS) != 0, pdis, par2.ro, par2.p);
                }
            } else if (ft == G_INNER_SPHERE) {
                par11 = par2;
            } else if (ft == G_AXIS) {
                par11.ro = par11.ro * sq(radius) / sq(dis);
                par11.Q = par11.Q * sq(radius) / sq(dis);
                par11.p = par11.p * (b.rp[c] / pow2g(dis, g2));
                polar_perenos(x, y, x2, y2, par11.u, par11.v);
                par2 = par11;
                par2.v = -par2.v;
                met = 0;
            }
            FluxOut<double> F;
            time = dmin_ref(time, P.kurant * dist / hllc_flux<TF>(P.gamma, P.kurant, par11, par2, 0.0, n1, n2, dist,
                                                                  met, false, F));
            Pt0 = Pt0 + F.P0 * S;
            Pt1 = Pt1 + F.P1 * S;
            Pt2 = Pt2 + F.P2 * S;
            Pt3 = Pt3 + F.P3 * S;
            Pt4 = Pt4 + F.PQ * S;
        }
        tmin_c = time;
        double q2_1, q2_2, q3;
        source_mk1(d, P, c, x, y, par1.u, par1.v, par1.ro, par1.p, q2_1, q2_2, q3, &status);
        const double ro = par1.ro, u = par1.u, v = par1.v, p = par1.p, Q = par1.Q;
        const double gm1 = P.gamma - 1;
        double ro3 = ro - dt * (Pt0 / Volume);
        const double Q33 = Q - (dt / Volume) * Pt4 - dt;
        if (ro3 <= 0) {
            ro3 = P.ro_floor;
            nro = 1;
        }
        const double u3 = (ro * u - dt * (Pt1 / Volume - q2_1)) / ro3;
        const double v3 = (ro * v - dt * ((Pt2 - p * 0.5 * (vs1 + vs2)) / Volume - q2_2)) / ro3;
        double p3 = (((p / gm1 + ro * (u * u + v * v) * 0.5) - dt * (Pt3 / Volume - q3)) - 0.5 * ro3 * (u3 * u3 + v3 * v3)) *
                    gm1;
        if (p3 <= 0) {
            p3 = P.p_floor;
            npc = 1;
        }
        b.nxt[0][c] = ro3;
        b.nxt[1][c] = p3;
        b.nxt[2][c] = u3;
        b.nxt[3][c] = v3;
        b.nxt[4][c] = Q33;
    }
    block_reduce_commit(tmin_c, nro, npc, status, b.dt_acc, b.counters, b.status);
}

// ------------------------------------------------------------------ inner form, four lanes per cell
// Go_stationary_5_komponent_inner_MK2 on a fixed grid with fixed Monte-Carlo
// moments: all a step needs beside the states is constant over a call, so one
// launch (inner_table_kernel) computes it per (cell, face) lane and the steps
// read it back: per lane i = 4 * (list position) + face, kInnerRows rows of
// 4 n_list doubles and kInnerIntRows rows of ints (type | flags, other cell,
// Sosed_down of either side).
//   0 n1, 1 n2, 2 S, 3 kurant * dist
//   4 kroO, 5 kpO, 6 CO, 7 SO   the cell's side: |centroid|^2 / |centre|^2,
//                               (|centroid| / |centre|)^(2 gamma), rotation
//                               to the face centre's polar frame
//   8 kroN, 9 kpN, 10 CN, 11 SN the other side's; Inner_sphere: wind ro, p, u, v
//   12 w1, 13 k1, 14 r12        radial TVD, the cell's side: factors of the
//                               Sosed_down cell's ro and p, 1 / (dist2 - dist1)
//   15 r23, 16 dist2            -1 / (dist2 + dist3) of both sides, distance
//   17 w1, 18 k1, 19 r12, 20 dist2  the same seen from the other side
//   21 uH, 22 vH, 23 roH, 24 th Monte-Carlo moments of species `face` at the
//                               cell, th = 2 pH / roH
//   25 k_u, k_v, k_T            of the cell, on its lanes 0, 1, 2
//   26 1 / Volume, 27 (vs1 + vs2) / 2   on lane 0
enum : int { IL_TYPE = 7, IL_TVD = 8, IL_RAW_O = 16, IL_RAW_N = 32, IL_SRC = 64, IL_ACT = 128 };

__global__ void __launch_bounds__(128) inner_table_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                          const int32_t* __restrict__ list, int n_list,
                                                          double* __restrict__ tab, int* __restrict__ itab) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t N = 4 * static_cast<size_t>(n_list);
    if (static_cast<size_t>(i) >= N) return;
    const int c = list[i >> 2], j = i & 3;
    double r[kInnerRows];
#pragma unroll
    for (int k = 0; k < kInnerRows; k++) r[k] = 0.0;
    int ft = IL_TYPE, flags = 0, nb = -1, sdO = c, sdN = c, status = 0;
    if (!(d.cflags[c] & CF_CENTR)) {
        flags = IL_ACT;
        const uint32_t cf = d.cflags[c];
        const int s0 = d.cstart[c], n = d.cstart[c + 1] - s0, g0 = d.gstart[c], g1 = d.gstart[c + 1];
        const int32_t* con = d.contour + s0;
        const double x = b.cx[c], y = b.cy[c], radius = sqrt(sq(x) + sq(y));
        if (j == 0) {
            r[26] = 1.0 / volume_rotate(con, n, d.X, d.Y);
            r[27] = 0.5 * (area(con, n, d.sA, d.sB, g0, g1, d.X, d.Y, false) +
                           area(con, n, d.sA, d.sB, g0, g1, d.X2, d.Y2, true));
        }
        const int g = g0 + j;
        if (g < g1) {
            const int A = d.sA[g], B = d.sB[g];
            ft = d.sinfo[g] & SI_TYPE_MASK;
            const double xa = d.X[A], ya = d.Y[A], xb = d.X[B], yb = d.Y[B];
            const double nn = sqrt(sq(xb - xa) + sq(yb - ya));
            const double x2 = (xa + xb) / 2.0, y2 = (ya + yb) / 2.0, dis2 = sq(x2) + sq(y2);
            const double dist = sqrt(sq(x - x2) + sq(y - y2));
            r[0] = (yb - ya) / nn;
            r[1] = -((xb - xa) / nn);
            r[2] = nn * (ya + yb) * 0.5;
            r[3] = P.kurant * dist;
            const double pdis = pow2g(sqrt(dis2), 2.0 * P.gamma);
            double cf2, sf2;
            polar_cs(x2, y2, cf2, sf2);
            auto side = [&](int k, double xc, double yc, double* o) {
                double c1, s1;
                polar_cs(xc, yc, c1, s1);
                o[0] = (sq(xc) + sq(yc)) / dis2;
                o[1] = b.rp[k] / pdis;
                o[2] = c1 * cf2 + s1 * sf2;
                o[3] = c1 * sf2 - s1 * cf2;
            };
            side(c, x, y, r + 4);
            if (ft == G_USUALY) {
                nb = d.snb[g];
                const double x3 = b.cx[nb], y3 = b.cy[nb], distn = sqrt(sq(x3 - x2) + sq(y3 - y2));
                side(nb, x3, y3, r + 8);
                const uint32_t nbf = d.cflags[nb];
                if ((cf & CF_C1) && (nbf & CF_C1)) {
                    flags |= IL_TVD;
                    r[15] = 1.0 / (-dist - distn);
                    // Get_par_TVD_radial of master M (centre xm, ym, distance dm)
                    auto tvd = [&](int M, double xm, double ym, double dm, int Sd, bool axis, const double* own,
                                   double* o, int& sd, int raw) {
                        sd = M;
                        if (Sd >= 0) {
                            const double xs = b.cx[Sd], ys = b.cy[Sd];
                            sd = Sd;
                            o[0] = (sq(xs) + sq(ys)) / dis2;
                            o[1] = b.rp[Sd] / pdis;
                            o[2] = 1.0 / (dm - sqrt(sq(x2 - xs) + sq(y2 - ys)));
                        } else if (axis) {  // the mirrored centre has the radius and state of M itself
                            o[0] = own[0];
                            o[1] = own[1];
                            o[2] = 1.0 / (dm - sqrt(sq(x2 - xm) + sq(y2 + ym)));
                        } else {
                            flags |= raw;
                        }
                    };
                    tvd(c, x, y, dist, d.ssd[g], (cf & CF_AXIS) != 0, r + 4, r + 12, sdO, IL_RAW_O);
                    r[16] = dist;
                    tvd(nb, x3, y3, distn, d.ssd2[g], (nbf & CF_AXIS) != 0, r + 8, r + 17, sdN, IL_RAW_N);
                    r[20] = distn;
                }
            } else if (ft == G_INNER_SPHERE) {
                const St5 w = inner_sphere_state(P, x2, y2);
                r[8] = w.ro;
                r[9] = w.p;
                r[10] = w.u;
                r[11] = w.v;
            }
        }
        const bool interp = radius > P.src_rmin && radius < P.src_rmax && x >= 0.0;
        int K_do = -1, K_posle = -1;
        if (!interp || source_bracket(d, c, radius, K_do, K_posle, &status)) {
            flags |= IL_SRC;
            SrcMoments m = source_moments(d, c, j, interp, K_do, K_posle, radius);
            if (m.roH <= 0.0) {
                m.roH = 0.0000001;
                m.pH = 0.0;
            }
            r[21] = m.uH;
            r[22] = m.vH;
            r[23] = m.roH;
            r[24] = 2.0 * m.pH / m.roH;
            r[25] = j == 0 ? m.ku : j == 1 ? m.kv : m.kT;
        }
    }
#pragma unroll
    for (int k = 0; k < kInnerRows; k++) tab[k * N + i] = r[k];
    itab[i] = ft | flags;
    itab[N + i] = nb;
    itab[2 * N + i] = sdO;
    itab[3 * N + i] = sdN;
    if (status) atomicOr(b.status, status);
}

// The steps of a call in one cooperative launch: a lane evaluates one face of
// its cell and one species' charge exchange, the cell's four lanes add both
// in the reference's order by shuffles, and one grid barrier ends the step
// (the CFL accumulators as in the plain form's kernels).  One thread per
// cell walking its faces (a pow and the radial reconstructions per face and
// side, 233 blocks) took 41.5 us per step on the 29.7k inner cells of the
// 200k grid, 12.1 us here.
template <typename TF>
__global__ void __launch_bounds__(256, 2) inner_lanes_kernel(DevMesh d, gelios_params P, StepBuffers b0, StepBuffers b1,
                                                             const int32_t* __restrict__ list, int n_list,
                                                             const double* __restrict__ tab,
                                                             const int* __restrict__ itab, int nsteps) {
    __shared__ double sm[32];
    cg::grid_group grid = cg::this_grid();
    const size_t N = 4 * static_cast<size_t>(n_list);
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    const int j = tid & 3, q0 = threadIdx.x & 28;
    const unsigned full = 0xffffffffu;
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    const double gm1 = P.gamma - 1, rg1 = 1.0 / gm1;
    const int rounds = static_cast<int>((N + nth - 1) / nth);
    double dt = *b0.dt_cur, dt_prev = dt;
    int nro = 0, npc = 0;
    for (int st = 0; st < nsteps; st++) {
        const StepBuffers& b = (st & 1) ? b1 : b0;
        double t = inf;
        for (int rd = 0; rd < rounds; rd++) {
            const size_t i = static_cast<size_t>(rd) * nth + tid;
            const bool in = i < N;
            const int c = in ? list[i >> 2] : 0;
            const int info = in ? itab[i] : IL_TYPE;
            const bool act = (info & IL_ACT) != 0;
            const int ft = info & IL_TYPE;
            const double* r = tab + i;
            St5 own{1.0, 1.0, 0.0, 0.0, 1.0};
            double F[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
            double nuu = 0.0, nuv = 0.0, nue = 0.0, kk = 0.0;
            if (act) {
                own = St5{__ldcg(b.cur[0] + c), __ldcg(b.cur[1] + c), __ldcg(b.cur[2] + c), __ldcg(b.cur[3] + c),
                          __ldcg(b.cur[4] + c)};
                t = dmin_ref(t, 10000000.0);
                if (info & IL_SRC) {
                    kk = r[25 * N];
                    source_rates_th(P, r[21 * N], r[22 * N], r[23 * N], r[24 * N], own.u, own.v, own.ro,
                                    own.p / own.ro, sq(own.u) + sq(own.v), nuu, nuv, nue);
                }
            }
            if (act && ft != IL_TYPE) {
                St5 L = own, R = own;
                const double n1 = r[0], n2 = r[N], S = r[2 * N];
                if (ft == G_USUALY) {
                    const int nb = itab[N + i];
                    R = St5{__ldcg(b.cur[0] + nb), __ldcg(b.cur[1] + nb), __ldcg(b.cur[2] + nb), __ldcg(b.cur[3] + nb),
                            __ldcg(b.cur[4] + nb)};
                    const double kO = r[4 * N], pO = r[5 * N], kN = r[8 * N], pN = r[9 * N];
                    const double roO = L.ro * kO, prO = L.p * pO, roN = R.ro * kN, prN = R.p * pN;
                    const double rawRo = R.ro, rawP = R.p;
                    L = plain_scale(L, kO, pO, r[6 * N], r[7 * N]);
                    R = plain_scale(R, kN, pN, r[10 * N], r[11 * N]);
                    L.Q *= kO;
                    R.Q *= kN;
                    if (info & IL_TVD) {
                        const int sO = itab[2 * N + i], sN = itab[3 * N + i];
                        const double r23 = r[15 * N];
                        const double o1 = __ldcg(b.cur[0] + sO), o2 = __ldcg(b.cur[1] + sO);
                        const double m1 = __ldcg(b.cur[0] + sN), m2 = __ldcg(b.cur[1] + sN);
                        const double rO = r[14 * N], dO = -r[16 * N], rN = r[19 * N], dN = -r[20 * N];
                        L.ro = linear3r(o1 * r[12 * N], roO, roN, rO, r23, dO);
                        L.p = linear3r(o2 * r[13 * N], prO, prN, rO, r23, dO);
                        R.ro = linear3r(m1 * r[17 * N], roN, roO, rN, r23, dN);
                        R.p = linear3r(m2 * r[18 * N], prN, prO, rN, r23, dN);
                        if (info & IL_RAW_O) {
                            L.ro = own.ro;
                            L.p = own.p;
                        }
                        if (info & IL_RAW_N) {
                            R.ro = rawRo;
                            R.p = rawP;
                        }
                    }
                } else if (ft == G_INNER_SPHERE) {
                    R = St5{r[8 * N], r[9 * N], r[10 * N], r[11 * N], r[8 * N]};
                    L = R;
                } else if (ft == G_AXIS) {
                    const double kO = r[4 * N];
                    L = plain_scale(L, kO, r[5 * N], r[6 * N], r[7 * N]);
                    L.Q *= kO;
                    R = L;
                    R.v = -R.v;
                } else if (ft == G_EXTERN) {
                    if (R.u >= 0.0) R.u = P.extern_u_par;
                } else if (ft == G_INPUT) {
                    R = input_state(P);
                }
                double UU;
                if (ft == G_AXIS) {  // HLL
                    FluxOut<double> G;
                    UU = hllc_flux<TF>(P.gamma, P.kurant, L, R, 0.0, n1, n2, 1.0, 0, false, G);
                    F[0] = G.P0;
                    F[1] = G.P1;
                    F[2] = G.P2;
                    F[3] = G.P3;
                    F[4] = G.PQ;
                } else {
                    UU = plain_flux<TF>(P, L, R, n1, n2, F);
                }
#pragma unroll
                for (int k = 0; k < 5; k++) F[k] *= S;
                t = dmin_ref(t, dt_candidate(r[3 * N] / UU));
            }
            double Pt[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, Mu = 0.0, Mv = 0.0, MT = 0.0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
#pragma unroll
                for (int f = 0; f < 5; f++) Pt[f] = Pt[f] + __shfl_sync(full, F[f], q0 + k);
                Mu = Mu + __shfl_sync(full, nuu, q0 + k);
                Mv = Mv + __shfl_sync(full, nuv, q0 + k);
                MT = MT + __shfl_sync(full, nue, q0 + k);
            }
            const double ku = __shfl_sync(full, kk, q0), kv = __shfl_sync(full, kk, q0 + 1),
                         kT = __shfl_sync(full, kk, q0 + 2);
            if (act && j == 0) {  // Setka.cpp:7167-7207
                const double q1 = P.src_coef * Mu * ku, q2 = P.src_coef * Mv * kv, q3 = P.src_coef * MT * kT;
                const double rV = r[26 * N], As = r[27 * N];
                const double ro = own.ro, u = own.u, v = own.v, p = own.p;
                double ro3 = ro - dt * (Pt[0] * rV);
                const double Q3 = own.Q - (dt * rV) * Pt[4] - dt;
                if (ro3 <= 0) {
                    ro3 = P.ro_floor;
                    nro++;
                }
                const double rro3 = 1.0 / ro3;
                const double u3 = (ro * u - dt * (Pt[1] * rV - q1)) * rro3;
                const double v3 = (ro * v - dt * ((Pt[2] - p * As) * rV - q2)) * rro3;
                double p3 = (((p * rg1 + ro * (u * u + v * v) * 0.5) - dt * (Pt[3] * rV - q3)) -
                             0.5 * ro3 * (u3 * u3 + v3 * v3)) *
                            gm1;
                if (p3 <= 0) {
                    p3 = P.p_floor;
                    npc++;
                }
                b.nxt[0][c] = ro3;
                b.nxt[1][c] = p3;
                b.nxt[2][c] = u3;
                b.nxt[3][c] = v3;
                b.nxt[4][c] = Q3;
            }
        }
        unsigned long long* acc = plain_acc(b0.dt_acc, st);
        t = block_min_nonneg(t, sm);
        if (threadIdx.x == 0 && t < inf) atomicMin(acc, static_cast<unsigned long long>(__double_as_longlong(t)));
        grid.sync();
        dt_prev = dt;
        dt = plain_dt(__ldcg(acc));
        if (tid == 0) *plain_acc(b0.dt_acc, st + 2) = 0x7ff0000000000000ULL;
    }
    if (nro) atomicAdd(&b0.counters[0], static_cast<unsigned long long>(nro));
    if (npc) atomicAdd(&b0.counters[1], static_cast<unsigned long long>(npc));
    if (tid == 0) {
        const StepBuffers& b = ((nsteps - 1) & 1) ? b1 : b0;
        *b.dt_next = dt;
        *const_cast<double*>(b.dt_cur) = dt_prev;
    }
}

// T[now2] of the reference: min(1e7, all face candidates) if any cell took
// part, 1e8 otherwise; re-arm the accumulator.
__global__ void dt_finalize_kernel(StepBuffers b) {
    const unsigned long long a = *b.dt_acc;
    double t = (a == 0x7ff0000000000000ULL) ? 100000000.0 : __longlong_as_double(static_cast<long long>(a));
    *b.dt_next = t;
    *b.dt_acc = 0x7ff0000000000000ULL;
}

// T[now2] when the update did not fold the 1e7 start of the CFL minimum in
// (the pipelined moving-grid step): a face candidate exists exactly when a
// cell takes part (a cell that takes part gives its faces a candidate), so
// min(1e7, candidates) if there is one, 1e8 otherwise; re-arm the
// accumulator.
__device__ __forceinline__ void dt_finalize_cap(const StepBuffers& b) {
    const unsigned long long a = *b.dt_acc;
    const double t = (a == 0x7ff0000000000000ULL)
                         ? 100000000.0
                         : dmin_ref(10000000.0, __longlong_as_double(static_cast<long long>(a)));
    *b.dt_next = t;
    *b.dt_acc = 0x7ff0000000000000ULL;
}

// x = x2, y = y2 (Setka.cpp:10473-10480; the zeroed V and count are never
// stored, see point_velocity) + dt finalisation (CAP: dt_finalize_cap).
template <bool CAP>
__global__ void commit_kernel(DevMesh d, StepBuffers b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        if (CAP) {
            dt_finalize_cap(b);
        } else {
            const unsigned long long a = *b.dt_acc;
            double t = (a == 0x7ff0000000000000ULL) ? 100000000.0 : __longlong_as_double(static_cast<long long>(a));
            *b.dt_next = t;
            *b.dt_acc = 0x7ff0000000000000ULL;
        }
    }
    if (i < d.n_points) {
        d.X[i] = d.X2[i];
        d.Y[i] = d.Y2[i];
    }
}

// ------------------------------------------------------------------ node velocities
// Move_surface, part 2 (Setka.cpp:3522-3535, 3718-3736, 3829-3842): the
// velocity of a tracked-surface node.  The reference accumulates the face
// speeds into Point::Vx/Vy/count in one serial pass per line, runs three
// averaging loops that all walk Line_Contact, and fixes up the end nodes of
// each line in between.  The three lines touch disjoint point sets, so the
// value of one node depends only on its own face incidences (sp_inc, in line
// order), on the averaging passes in which it is the A end of a contact face
// (sp_ainc), and, for the end nodes, on the first-pass values of the other
// end nodes of its line.  point_velocity replays exactly those operations for
// one point, so the rails can evaluate their key points directly from the
// per-face speeds (bit-identical to the serial passes).
__device__ __forceinline__ void node_pass1(const DevMesh& d, const double* __restrict__ scratch, int i, int line,
                                           double& v, double& w, int& c) {
    // the node's faces and their rows, each in one level of loads
    const int4 inc = reinterpret_cast<const int4*>(d.sp_inc)[i];
    const int e[4] = {inc.x, inc.y, inc.z, inc.w};
    const int4 ai = reinterpret_cast<const int4*>(d.sp_ainc)[i];
    const int an[4] = {ai.x, ai.y, ai.z, ai.w};
    double2 f01[4], f23[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double2* r = reinterpret_cast<const double2*>(scratch + 4 * (e[k] < 0 ? 0 : e[k] >> 1));
        f01[k] = r[0];
        f23[k] = r[1];
    }
    v = 0.0;
    w = 0.0;
    c = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (e[k] < 0) break;
        const int role = e[k] & 1;  // role 0: A end, 1: B end
        const double f[4] = {f01[k].x, f01[k].y, f23[k].x, f23[k].y};
        const double br = f[3];
        bool add;
        if (line == 0) add = role == 1;
        else if (line == 1) add = role == 1 || br != 0.0;
        else add = (br == 1.0) || (role == 1 && (br == 0.0 || br == 2.0)) || (role == 0 && br == 3.0);
        if (add) {
            v += f[0] * f[1];
            w += f[0] * f[2];
            c++;
        }
    }
    if (line == 0) {  // first averaging pass: every contact face (Setka.cpp:3522-3530)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (an[k] < 0) break;
            if (c > 0) {
                v /= (1.0 * c);
                w /= (1.0 * c);
            }
        }
    }
}

// Vx, Vy after Move_surface of the node i of each group of eight lanes (0 for
// i < 0, a point off the tracked lines: every step starts from zero
// velocities, Setka.cpp:10473-10480), called by a whole warp.  Lane 4 of the
// group takes the node's own first pass, lanes 0-3 those of the four end
// nodes of its line when the node is one of them; every lane gets the result.
__device__ __forceinline__ void point_velocity(const DevMesh& d, const double* __restrict__ scratch, double dt, int i,
                                               double& vx, double& vy) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, m = lane & 7, g0 = lane & 24;
    const int line = i >= 0 ? d.sp_line[i] : 0;
    const int4 fx = reinterpret_cast<const int4*>(d.sp_fix)[line];  // a0, b0 (first face), a_last, b_last
    const bool end = i >= 0 && (i == fx.x || i == fx.w);
    const int own = m == 0 ? fx.x : m == 1 ? fx.y : m == 2 ? fx.z : fx.w;
    const int node = m == 4 ? i : (end && m < 4) ? own : -1;
    double v = 0.0, w = 0.0, px = 0.0, py = 0.0;
    int c = 0;
    if (node >= 0) {
        if (end) {
            const int p = d.sp_point[node];
            px = d.X[p];
            py = d.Y[p];
        }
        node_pass1(d, scratch, node, line, v, w, c);
    }
    double lx[4], ly[4], ex[4], ey[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        lx[q] = __shfl_sync(full, v, g0 + q);
        ly[q] = __shfl_sync(full, w, g0 + q);
        ex[q] = __shfl_sync(full, px, g0 + q);
        ey[q] = __shfl_sync(full, py, g0 + q);
    }
    vx = __shfl_sync(full, v, g0 + 4);
    vy = __shfl_sync(full, w, g0 + 4);
    c = __shfl_sync(full, c, g0 + 4);
    if (i < 0) return;
    if (end) {
        // replay the end-node fix-ups of this line in the reference's order
        // on local copies of the four end nodes (aliases kept in sync)
        const int id[4] = {fx.x, fx.y, fx.z, fx.w};
        auto setx = [&](int nd, double val) {
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (id[q] == nd) lx[q] = val;
        };
        auto sety = [&](int nd, double val) {
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (id[q] == nd) ly[q] = val;
        };
        // fx[0]: vx[a0] = vx[b0] + (X[b0] - X[a0]) / dt on every line
        setx(id[0], lx[1] + (ex[1] - ex[0]) / dt);
        if (line == 1) {
            // inner shock: vx[b1] = vx[a1] + (X[a1] - X[b1]) / dt (Setka.cpp:3733-3736)
            double a1x = lx[2];
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (id[q] == id[2]) a1x = lx[q];
            setx(id[3], a1x + (ex[2] - ex[3]) / dt);
        } else {
            // contact / outer shock: vy[b1] = vy[a1] + (Y[a1] - Y[b1]) / dt
            sety(id[3], ly[2] + (ey[2] - ey[3]) / dt);
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (id[q] == i) {
                vx = lx[q];
                vy = ly[q];
            }
    }
    if (line == 0) {
        // second and third passes walk Line_Contact up to the inner/outer
        // line lengths (Setka.cpp:3718-3731, 3829-3837)
        const int nC = d.n_lc, nI = d.n_li, nO = d.n_lo;
        const int lim2 = nI > 0 ? (nI < nC ? nI : nC) : 0;
        const int lim3 = nO > 0 ? (nO < nC ? nO : nC) : 0;
        const int4 ai = reinterpret_cast<const int4*>(d.sp_ainc)[i];
        const int an[4] = {ai.x, ai.y, ai.z, ai.w};
        for (int pass = 0; pass < 2; pass++) {
            const int lim = pass == 0 ? lim2 : lim3;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int j = an[k];
                if (j < 0) break;
                if (j < lim && c > 0) {
                    vx /= (1.0 * c);
                    vy /= (1.0 * c);
                }
            }
        }
    }
}

// ------------------------------------------------------------------ grid motion
// Move_Setka_Calculate_2 (Setka.cpp:4324-4759) in one launch, one CTA per
// rail.  The reference moves the A rails, then the B rails, then the C rails,
// then the D rails, and two of them share points:
//  * C_Rails[0] starts with the first M1 points of the last B rail and
//    overwrites them (with its own angle), so the last B rail leaves those
//    points to C_Rails[0] and uses its own value of its key point 0 for the
//    points above it, as the reference's B pass does;
//  * the first point of every D rail is a point of C_Rails[0]; the D block
//    recomputes that point's new position from C_Rails[0]'s key point with
//    the same operations (bit-identical to reading it back).
// The rails' constants: cos and sin of their angle, and of every point the
// power law its radius or height follows between two key points (inner layer,
// Setka.cpp:4390-4406; the A rails' outer layer, 4443-4456).
__global__ void rail_table_kernel(DevMesh d, int ni, double* __restrict__ rcs, double* __restrict__ rsn,
                                  double* __restrict__ rfrac) {
    const int q = blockIdx.x;
    const double s = d.rs[q];
    if (threadIdx.x == 0) {
        rcs[q] = cos(s);
        rsn[q] = sin(s);
    }
    const int t = d.rtype[q], p0 = d.rpstart[q], np = d.rpstart[q + 1] - p0;
    const int M1 = d.rM[4 * q], M2 = d.rM[4 * q + 1], M3 = d.rM[4 * q + 2], M4 = d.rM[4 * q + 3];
    const double dd = 1.5708 / sqrt(1.0 - 1.0 / 1.76);
    const double e = 1.76 * (1.0 - sq(s / dd));
    for (int j = threadIdx.x; j < np; j += blockDim.x) {
        double f = 0.0;
        if (t <= 2 && j < M1 - 1) {
            if (j < ni) {
                const double x = j * 1.0 / (ni);
                f = pow(x, 1.3);
            } else {
                const double x = (j - ni) * 1.0 / (M1 - 1 - ni);
                f = pow(x, 1.05);
            }
        } else if (t == 0 && j >= M1 + M2 + M3) {
            const double x = (j - (M1 + M2 + M3) + 1) * 1.0 / (M4);
            f = pow(x, e);
        }
        rfrac[p0 + j] = f;
    }
}

// copy_outer_shock: Move_Setka_Calculate_2 gives the D rails beyond
// n_outer_shock the outer-shock key height of the last D rail before them
// (Setka.cpp:4725-4728); Move_Setka_Calculate (Setka.cpp:4761-5147, used by
// Go_5_komponent) is otherwise the same and moves them on their own.
// One rail q (the body of rails_kernel; every thread of the block calls it).
__device__ __forceinline__ void rails_body(const DevMesh& d, const gelios_params& P, const double* __restrict__ dtp,
                                           const double* __restrict__ scratch, bool copy_outer_shock, int q) {
    const double dt = *dtp;
    const int32_t* ap = d.rpts + d.rpstart[q];
    const int np = d.rpstart[q + 1] - d.rpstart[q];
    const int32_t* kp = d.rkeys + d.rkstart[q];
    const int M1 = d.rM[4 * q], M2 = d.rM[4 * q + 1], M3 = d.rM[4 * q + 2], M4 = d.rM[4 * q + 3];
    const int t = d.rtype[q];
    const int first_c = d.n_rail_a + d.n_rail_b, first_d = first_c + d.n_rail_c;
    // the last B rail hands its first M1 points to C_Rails[0]
    const bool handoff = (t == 1) && (q == first_c - 1) && d.n_rail_c > 0;
    double* X2 = d.X2;
    double* Y2 = d.Y2;
    const double* X = d.X;
    const double* Y = d.Y;
    __shared__ double sh[6];
    const int ni = P.n_inner;
    // velocities and positions of the key points this rail reads, by the
    // first warp, eight lanes a point
    __shared__ double kvx[4], kvy[4], kx[4], ky[4];
    const double* frac = d.rfrac + d.rpstart[q];
    const int K3 = t == 2 ? -1 : kp[3];
    double x3 = 0.0, y3 = 0.0;
    if (threadIdx.x == 0 && K3 >= 0) {
        x3 = X[K3];
        y3 = Y[K3];
    }
    if (threadIdx.x < 32) {
        const int k = threadIdx.x >> 3;
        const int4 pp = d.rk_point[q], nn = d.rk_node[q];
        int pt = k == 0 ? pp.x : k == 1 ? pp.y : k == 2 ? pp.z : -1;
        int node = k == 0 ? nn.x : k == 1 ? nn.y : k == 2 ? nn.z : -1;
        if (k == 3 && t == 3 && copy_outer_shock && q - first_d >= P.n_outer_shock && P.n_outer_shock >= 1) {
            pt = d.rkeys[d.rkstart[first_d + P.n_outer_shock - 1] + 2];
            node = d.sp_of_point[pt];
        }
        double xp = 0.0, yp = 0.0;
        if (pt >= 0) {
            xp = X[pt];
            yp = Y[pt];
        }
        double vx, vy;
        point_velocity(d, scratch, dt, node, vx, vy);
        if ((threadIdx.x & 7) == 0) {
            kvx[k] = vx;
            kvy[k] = vy;
            kx[k] = xp;
            ky[k] = yp;
        }
    }
    __syncthreads();
    if (t == 0 || t == 1 || t == 2) {
        const double cs = d.rcs[q], sn = d.rsn[q];
        if (threadIdx.x == 0) {
            if (t == 0) {  // A rail, Setka.cpp:4331-4356
                for (int kk = 0; kk < 3; kk++) {
                    const int K = kp[kk];
                    const double V = kvx[kk] * cs + kvy[kk] * sn;
                    X2[K] = kx[kk] + dt * V * cs;
                    Y2[K] = ky[kk] + dt * V * sn;
                }
                X2[K3] = x3;
                Y2[K3] = y3;
                sh[0] = sqrt(sq(X2[kp[0]]) + sq(Y2[kp[0]]));
                sh[1] = sqrt(sq(X2[kp[1]]) + sq(Y2[kp[1]]));
                sh[2] = sqrt(sq(X2[kp[2]]) + sq(Y2[kp[2]]));
            } else if (t == 1) {  // B rail, Setka.cpp:4469-4502
                const int K0 = kp[0], K1 = kp[1], K2 = kp[2];
                double V = kvx[0] * cs + kvy[0] * sn;
                const double x0 = kx[0] + dt * V * cs, y0 = ky[0] + dt * V * sn;
                if (!handoff) {
                    X2[K0] = x0;
                    Y2[K0] = y0;
                }
                V = kvx[1] * 0.0 + kvy[1] * 1.0;
                X2[K1] = x0;
                Y2[K1] = ky[1] + dt * V;
                V = kvx[2] * 0.0 + kvy[2] * 1.0;
                X2[K2] = x0;
                Y2[K2] = ky[2] + dt * V;
                X2[K3] = x0;
                Y2[K3] = y3;
                sh[0] = sqrt(sq(x0) + sq(y0));
                sh[1] = Y2[K1];
                sh[2] = Y2[K2];
                sh[3] = x0;
                sh[4] = y0;
            } else {  // C rail, Setka.cpp:4603-4614
                const int K0 = kp[0], K1 = kp[1];
                const double V = kvx[0] * cs + kvy[0] * sn;
                X2[K0] = kx[0] + dt * V * cs;
                Y2[K0] = ky[0] + dt * V * sn;
                X2[K1] = P.Left;
                Y2[K1] = Y[K1];
                sh[0] = sqrt(sq(X2[K0]) + sq(Y2[K0]));
                sh[3] = X2[K0];
                sh[4] = Y2[K0];
            }
        }
        __syncthreads();
        const double R2 = sh[0];
        if (!handoff) {  // inner layer, Setka.cpp:4390-4406 (and 4532-4548, 4644-4660)
            for (int j = threadIdx.x; j < M1 - 1; j += blockDim.x) {
                double r;
                if (j < ni) r = P.R1 + frac[j] * (P.R111 - P.R1);
                else r = P.R111 + frac[j] * (R2 - P.R111);
                X2[ap[j]] = r * cs;
                Y2[ap[j]] = r * sn;
            }
        }
        if (t == 0) {  // Setka.cpp:4411-4456
            const double R3 = sh[1], R4 = sh[2];
            for (int j = threadIdx.x; j < M2 - 1; j += blockDim.x) {
                const double r = R2 + (R3 - R2) * (j + 1) / (M2);
                X2[ap[M1 + j]] = r * cs;
                Y2[ap[M1 + j]] = r * sn;
            }
            for (int j = threadIdx.x; j < M3 - 1; j += blockDim.x) {
                const double r = R3 + (R4 - R3) * (j + 1) / (M3);
                X2[ap[M1 + M2 + j]] = r * cs;
                Y2[ap[M1 + M2 + j]] = r * sn;
            }
            for (int j = threadIdx.x; j < M4; j += blockDim.x) {
                const double r = R4 + frac[M1 + M2 + M3 + j] * (P.R5 - R4);
                X2[ap[M1 + M2 + M3 + j]] = r * cs;
                Y2[ap[M1 + M2 + M3 + j]] = r * sn;
            }
        } else if (t == 1) {  // Setka.cpp:4552-4593
            const double R2y = sh[4], R3 = sh[1], R4 = sh[2], xk = sh[3];
            for (int j = threadIdx.x; j < M2 - 1; j += blockDim.x) {
                X2[ap[M1 + j]] = xk;
                Y2[ap[M1 + j]] = R2y + (R3 - R2y) * (j + 1) / (M2);
            }
            for (int j = threadIdx.x; j < M3 - 1; j += blockDim.x) {
                X2[ap[M1 + M2 + j]] = xk;
                Y2[ap[M1 + M2 + j]] = R3 + (R4 - R3) * (j + 1) / (M3);
            }
            for (int j = threadIdx.x; j < M4; j += blockDim.x) {
                X2[ap[M1 + M2 + M3 + j]] = xk;
                Y2[ap[M1 + M2 + M3 + j]] = R4 + (P.R5 - R4) * (j + 1) / (M4);
            }
        } else {  // Setka.cpp:4662-4673
            const double R2x = sh[3], yk = sh[4];
            const double x = pow(P.Left / (R2x), 1.0 / (M2));
            for (int j = M1 + threadIdx.x; j < np; j += blockDim.x) {
                X2[ap[j]] = R2x * pow(x, static_cast<double>(j + 1 - M1));
                Y2[ap[j]] = yk;
            }
        }
        return;
    }
    // D rail, Setka.cpp:4676-4758
    const int jj = q - first_d;
    const int sM2 = d.dims[5], sM3 = d.dims[6], sM4 = d.dims[7];
    if (threadIdx.x == 0) {
        const int K1 = kp[1], K2 = kp[2];
        // key point 0 = point M1 + jj of C_Rails[0], as the C pass moves it
        const double cs = d.rcs[first_c], sn = d.rsn[first_c];
        const double V0 = kvx[0] * cs + kvy[0] * sn;
        const double c0x = kx[0] + dt * V0 * cs, c0y = ky[0] + dt * V0 * sn;
        const int Mc1 = d.rM[4 * first_c], Mc2 = d.rM[4 * first_c + 1];
        const int j = Mc1 + jj;
        const double xr = pow(P.Left / (c0x), 1.0 / (Mc2));
        const double x0 = c0x * pow(xr, static_cast<double>(j + 1 - Mc1));
        const double y0 = c0y;
        double V = kvy[1];
        X2[K1] = x0;
        Y2[K1] = ky[1] + dt * V;
        V = kvy[2];
        X2[K2] = x0;
        if (copy_outer_shock && jj >= P.n_outer_shock && P.n_outer_shock >= 1) {
            Y2[K2] = ky[3] + dt * kvy[3];
        } else {
            Y2[K2] = ky[2] + dt * V;
        }
        X2[K3] = x0;
        Y2[K3] = y3;
        sh[0] = y0;
        sh[1] = Y2[K1];
        sh[2] = Y2[K2];
        sh[3] = x0;
    }
    __syncthreads();
    const double R2 = sh[0], R3 = sh[1], R4 = sh[2], xk = sh[3];
    for (int j = threadIdx.x; j < sM2 - 1; j += blockDim.x) {
        X2[ap[j + 1]] = xk;
        Y2[ap[j + 1]] = R2 + (R3 - R2) * (j + 1) / (M2);
    }
    for (int j = threadIdx.x; j < sM3 - 1; j += blockDim.x) {
        X2[ap[sM2 + j + 1]] = xk;
        Y2[ap[sM2 + j + 1]] = R3 + (R4 - R3) * (j + 1) / (M3);
    }
    for (int j = threadIdx.x; j < sM4; j += blockDim.x) {
        X2[ap[sM2 + sM3 + j + 1]] = xk;
        Y2[ap[sM2 + sM3 + j + 1]] = R4 + (P.R5 - R4) * (j + 1) / (M4);
    }
}

__global__ void __launch_bounds__(128) rails_kernel(DevMesh d, gelios_params P, const double* __restrict__ dtp,
                                                    const double* __restrict__ scratch, bool copy_outer_shock) {
    rails_body(d, P, dtp, scratch, copy_outer_shock, blockIdx.x);
}

// ------------------------------------------------------------------ surface tracking
// Get_par_TVD of a tracked face with end points a, bb seen from master M.
__device__ St5 face_tvd(const DevMesh& d, const double* const* st, const double* cx, const double* cy, int a, int bb,
                        int ft, int M, int So, int Sd, bool axis, bool tracked, int* status) {
    const double fx = (d.X[a] + d.X[bb]) / 2.0, fy = (d.Y[a] + d.Y[bb]) / 2.0;
    const St5 Ms = load_state(st, M);
    if (ft == G_USUALY) return tvd_usualy(st, cx, cy, fx, fy, Ms, cx[M], cy[M], So, Sd, axis, tracked, status);
    if (ft == G_AXIS) return tvd_axis(st, cx, cy, fx, fy, Ms, cx[M], cy[M], Sd);
    St5 o = Ms;
    return o;  // Extern/Upper_wall/Input/Inner faces do not occur on tracked lines
}

// Move_surface (Setka.cpp:3378-3844), part 1: one thread per tracked face
// (contact, inner shock, outer shock) computes its exact-Godunov wave speed,
// the face normal and the branch the reference takes.
// scratch layout per face j of the concatenated lines (contact, inner, outer):
//   [0] speed  [1] n1  [2] n2  [3] branch
//   branch: contact 0 (B only); inner 0 (B only) / 1 (A and B);
//           outer -1 (skipped) / 0 B / 1 A and B / 2 B / 3 A
// One warp per face: the lanes hold identical copies of the face's data, the
// exact solver runs warp-cooperatively, lane 0 writes.
// Tracked face j of the concatenated lines, all 32 lanes of a warp (the
// body of surface_faces_kernel).
__device__ __forceinline__ void surface_face_body(const DevMesh& d, const gelios_params& P, const StepBuffers& b,
                                                  double* __restrict__ scratch, int j, int lane) {
    const int nC = d.n_lc, nI = d.n_li;
    const double* const* st = b.cur;
    int status = 0;
    const double ga = P.gamma, g2 = 2.0 * P.gamma;
    double nv[3], q1[5], q2[5], qq[5], ds[3];
    const int4 r0 = d.sf_rec[3 * j], r1 = d.sf_rec[3 * j + 1];
    const int fl = d.sf_rec[3 * j + 2].x;
    const int a = r0.x, bb = r0.y;
    const bool trk = (fl & SF_TRACKED) != 0;
    // the face as its copy's master sees it
    auto tvd_copy = [&]() {
        return face_tvd(d, st, b.cx, b.cy, a, bb, (fl >> SF_TYPE2) & 7, r1.y, r1.z, r1.w, (fl & SF_AXIS2) != 0, trk,
                        &status);
    };
    double t1 = d.X[bb] - d.X[a], t2 = d.Y[bb] - d.Y[a];
    const double nn = sqrt(sq(t1) + sq(t2));
    t1 /= nn;
    t2 /= nn;
    const double n1 = t2, n2 = -t1;
    nv[0] = n1; nv[1] = n2; nv[2] = 0.0;
    double o0 = 0.0, o3 = 0.0;
    // TVD states of the face (even lanes) and of its twin (odd lanes),
    // exchanged between lane pairs
    auto tvd_pair = [&](St5& pf, St5& pc) {
        const bool cp = lane & 1;
        const St5 mine = face_tvd(d, st, b.cx, b.cy, a, bb, (cp ? fl >> SF_TYPE2 : fl) & 7, cp ? r1.y : r0.z,
                                  cp ? r1.z : r0.w, cp ? r1.w : r1.x, (fl & (cp ? SF_AXIS2 : SF_AXIS1)) != 0, trk,
                                  &status);
        St5 other;
        other.ro = __shfl_xor_sync(0xffffffffu, mine.ro, 1);
        other.p = __shfl_xor_sync(0xffffffffu, mine.p, 1);
        other.u = __shfl_xor_sync(0xffffffffu, mine.u, 1);
        other.v = __shfl_xor_sync(0xffffffffu, mine.v, 1);
        other.Q = __shfl_xor_sync(0xffffffffu, mine.Q, 1);
        pf = (lane & 1) ? other : mine;
        pc = (lane & 1) ? mine : other;
    };
    if (j < nC) {
        St5 p1, p2;
        tvd_pair(p1, p2);
        q1[0] = p1.ro; q1[1] = p1.p; q1[2] = p1.u; q1[3] = p1.v; q1[4] = 0.0;
        q2[0] = p2.ro; q2[1] = p2.p; q2[2] = p2.u; q2[3] = p2.v; q2[4] = 0.0;
        godunov_dev<true>(ga, P.kurant, q1, q2, nv, qq, ds, 0.0, 0.0, P.godunov_max_iter, &status, nullptr,
                          nullptr, true);
        o0 = ds[2] * P.koef * 0.3;
        o3 = 0.0;
    } else if (j < nC + nI) {
        const int M = r0.z;
        St5 p1 = load_state(st, M);
        const double x = b.cx[M], y = b.cy[M];
        const double radius = sqrt(sq(x) + sq(y));
        const double x2 = (d.X[a] + d.X[bb]) / 2.0, y2 = (d.Y[a] + d.Y[bb]) / 2.0;
        const double dis = sqrt(sq(x2) + sq(y2));
        const St5 p2 = tvd_copy();
        p1.ro = p1.ro * sq(radius) / sq(dis);
        p1.p = p1.p * (b.rp[M] / pow2g(dis, g2));
        polar_perenos(x, y, x2, y2, p1.u, p1.v);
        q1[0] = p1.ro; q1[1] = p1.p; q1[2] = p1.u; q1[3] = p1.v; q1[4] = 0.0;
        q2[0] = p2.ro; q2[1] = p2.p; q2[2] = p2.u; q2[3] = p2.v; q2[4] = 0.0;
        godunov_dev<true>(ga, P.kurant, q1, q2, nv, qq, ds, 0.0, 0.0, P.godunov_max_iter, &status, nullptr,
                          nullptr, true);
        o0 = ds[0] * P.koef * 0.1;
        const double tt1 = -n2, tt2 = n1;
        o3 = (fabs(p2.u * tt1 + p2.v * tt2) < 0.1) ? 1.0 : 0.0;
    } else {
        const int jj = j - nC - nI;
        const int lim = P.n_outer_shock + d.dims[0] + d.dims[1] + 1;
        if (jj >= lim) {
            o0 = 0.0;
            o3 = -1.0;
        } else {
            St5 p1, p2;
            tvd_pair(p1, p2);
            q1[0] = p1.ro; q1[1] = p1.p; q1[2] = p1.u; q1[3] = p1.v; q1[4] = 0.0;
            q2[0] = p2.ro; q2[1] = p2.p; q2[2] = p2.u; q2[3] = p2.v; q2[4] = 0.0;
            godunov_dev<true>(ga, P.kurant, q1, q2, nv, qq, ds, 0.0, 0.0, P.godunov_max_iter, &status, nullptr,
                          nullptr, true);
            o0 = ds[1] * P.koef;
            const double tt1 = -n2, tt2 = n1;
            double br;
            if ((sq(p1.u) + sq(p1.v) + sq(0.0)) / (ga * p1.p / p1.ro) > 1.0) br = 0.0;
            else if (fabs(p1.u * tt1 + p1.v * tt2) < 0.01) br = 1.0;
            else if (p1.u * tt1 + p1.v * tt2 > 0) br = 2.0;
            else br = 3.0;
            o3 = br;
        }
    }
    status = static_cast<int>(__reduce_or_sync(0xffffffffu, static_cast<unsigned>(status)));
    if (lane == 0) {
        double* out = scratch + 4 * j;
        out[0] = o0;
        out[1] = n1;
        out[2] = n2;
        out[3] = o3;
        if (status) atomicOr(b.status, status);
    }
}

// fin: finalise the step's dt first (fb: the buffers of the step before), for
// a call whose steps follow one another without a commit; nothing here reads
// it, the rails do.
__global__ void __launch_bounds__(64) surface_faces_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                           double* __restrict__ scratch, StepBuffers fb, bool fin) {
    if (fin && blockIdx.x == 0 && threadIdx.x == 0) dt_finalize_cap(fb);
    const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (j >= d.n_lc + d.n_li + d.n_lo) return;
    surface_face_body(d, P, b, scratch, j, threadIdx.x & 31);
}

// ------------------------------------------------------------------ per-face batches (known-answer checks)
__global__ void hllc_batch_kernel(gelios_params P, int n, const double* __restrict__ in, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* a = in + 16 * i;
    St5 L, R;
    L.ro = a[0]; L.Q = a[1]; L.p = a[2]; L.u = a[3]; L.v = a[4];
    R.ro = a[5]; R.Q = a[6]; R.p = a[7]; R.u = a[8]; R.v = a[9];
    FluxOut<double> F;
    double t;
    if (P.precision == GELIOS_PREC_FP32_FLUX)
        t = hllc_flux<float>(P.gamma, P.kurant, L, R, a[10], a[11], a[12], a[13], (int)a[14], a[15] != 0.0, F);
    else if (P.precision == GELIOS_PREC_FP32_WAVES)
        t = hllc_flux<WaveF32>(P.gamma, P.kurant, L, R, a[10], a[11], a[12], a[13], (int)a[14], a[15] != 0.0, F);
    else
        t = hllc_flux<double>(P.gamma, P.kurant, L, R, a[10], a[11], a[12], a[13], (int)a[14], a[15] != 0.0, F);
    t = P.kurant * a[13] / t;
    double* o = out + 9 * i;
    o[0] = t;
    o[1] = F.P0;
    o[2] = F.P1;
    o[3] = F.P2;
    o[4] = F.P3;
    o[5] = F.PQ;
    // wave speeds (Vl, Vc, Vp) recomputed in FP64 for the check
    const double n1 = a[11], n2 = a[12];
    const double u1 = L.u * n1 + L.v * n2, u2 = R.u * n1 + R.v * n2;
    const double cL = sqrt(P.gamma * L.p / L.ro), cR = sqrt(P.gamma * R.p / R.ro);
    const double SL = dmin_ref(u1, u2) - dmax_ref(cL, cR);
    const double SR = dmax_ref(u1, u2) + dmax_ref(cL, cR);
    const double suR = SR - u2, suL = SL - u1;
    o[6] = SL;
    o[7] = (suR * R.ro * u2 - suL * L.ro * u1 - R.p + L.p) / (suR * R.ro - suL * L.ro);
    o[8] = SR;
}

// One warp per problem (the warp-cooperative solver of the step kernels).
__global__ void godunov_batch_kernel(gelios_params P, int n, const double* __restrict__ in, double* __restrict__ out) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= n) return;
    const double* a = in + 15 * i;
    double q1[5], q2[5], nv[3], qq[5], ds[3];
    for (int k = 0; k < 5; k++) {
        q1[k] = a[k];
        q2[k] = a[5 + k];
    }
    nv[0] = a[10]; nv[1] = a[11]; nv[2] = a[12];
    int status = 0;
    const double t = P.kurant * a[14] / godunov_dev<true>(P.gamma, P.kurant, q1, q2, nv, qq, ds, a[13], a[14],
                                                          P.godunov_max_iter, &status);
    if ((threadIdx.x & 31) != 0) return;
    double* o = out + 10 * i;
    o[0] = t;
    for (int k = 0; k < 5; k++) o[1 + k] = qq[k];
    o[6] = ds[0];
    o[7] = ds[1];
    o[8] = ds[2];
    o[9] = status;
}

// HLLDQ_Korolkov batch: in[23] = L[9], R[9], n[3], rad, metod; out[10] =
// time, P[8], PQ.
__global__ void hlldq_batch_kernel(gelios_params P, int n, const double* __restrict__ in, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* a = in + 23 * i;
    double L[9], R[9], Po[8], PQ = 0.0;
    for (int k = 0; k < 9; k++) {
        L[k] = a[k];
        R[k] = a[9 + k];
    }
    for (int k = 0; k < 8; k++) Po[k] = 0.0;
    const double t = hlldq_korolkov(P.gamma, P.kurant, L, R, a[18], a[19], a[20], a[21], static_cast<int>(a[22]),
                                    Po, &PQ);
    double* o = out + 10 * i;
    o[0] = t;
    for (int k = 0; k < 8; k++) o[1 + k] = Po[k];
    o[9] = PQ;
}

// HLLD_Solver_Alexashov batch: in[21] = q1[8], q2[8], n[3], w, dist; out[13]
// = time, q[8], dsl, dsp, dsc, status.
__global__ void hlld_batch_kernel(gelios_params P, int n, const double* __restrict__ in, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* a = in + 21 * i;
    double q1[8], q2[8], nv[3], q[8], ds[3];
    for (int k = 0; k < 8; k++) {
        q1[k] = a[k];
        q2[k] = a[8 + k];
    }
    nv[0] = a[16];
    nv[1] = a[17];
    nv[2] = a[18];
    int status = 0;
    const double t = hlld_alexashov(P.gamma, P.kurant, q1, q2, nv, q, ds, a[19], a[20], &status);
    double* o = out + 13 * i;
    o[0] = t;
    for (int k = 0; k < 8; k++) o[1 + k] = q[k];
    o[9] = ds[0];
    o[10] = ds[1];
    o[11] = ds[2];
    o[12] = status;
}

// ------------------------------------------------------------------ four hydrogen fluids
// Setka::Go_5_komponent (Setka.cpp:8269-8950): the plasma and four hydrogen
// fluids H1..H4, each with its own HLLC flux, on the grid moved by
// Move_surface + Move_Setka_Calculate.  The 21-field state follows the
// member order of Parametr's aggregate initialisers (Gran.cpp:262-265):
// ro, p, u, v, Q, then ro, p, u, v of H1..H4.
constexpr double kNHOverKn = 1.0 / 6.0;   // n_H_LISM_ / Kn_, Help.h:60, 65

// The state rows of the five fluids: fluid 0 the plasma (with Q), 1..4 the
// hydrogen fluids H1..H4 (Q = the plasma's, which their flux ignores).
struct K5Rows {
    const double* const* st;
    const double* hs;
    size_t nc;
    __device__ __forceinline__ St5 load(int f, int c) const {
        if (f == 0) return load_state(st, c);
        const double* h = hs + static_cast<size_t>(4 * (f - 1)) * nc + c;
        return St5{h[0], h[nc], h[2 * nc], h[3 * nc], 0.0};
    }
};

// What the reconstruction of one side of a face needs of the grid, the same
// for the five fluids.  M the side's cell, So the other one, Sd Sosed_down.
struct K5Side {
    int M, Sd;
    bool axis, c1;
    double dM, dS, r12;        // face centre to M and So, 1 / (dM - d(Sd))
    double dm;                 // to the mirror image of M (axis cells without Sd)
    // C_1 cells: |M|^2 / |f|^2, (|M| / |f|)^(2 gamma), sqrt(|M| / |f|), the
    // same of So (S) and Sd (D), and the rotation to the face centre's frame
    double kro, kp, kh, kroS, kpS, khS, kroD, kpD, khD, C, Sn;
};
template <int GROUP>
__device__ __forceinline__ K5Side k5_side(const StepBuffers& b, int M, double xm, double ym, int So, double xs,
                                          double ys, int Sd, uint32_t mf, double x2, double y2, double dM, double dS,
                                          double dis2, double pdis, double cf, double sf) {
    K5Side s;
    s.M = M;
    s.Sd = Sd;
    s.axis = (mf & CF_AXIS) != 0;
    s.c1 = GROUP != kPlainGroup && (mf & CF_C1);
    s.dM = dM;
    s.dS = dS;
    s.r12 = s.dm = 0.0;
    double xd = 0.0, yd = 0.0;
    if (Sd >= 0) {
        xd = b.cx[Sd];
        yd = b.cy[Sd];
        s.r12 = 1.0 / (dM - sqrt(sq(x2 - xd) + sq(y2 - yd)));
    } else if (s.axis) {
        s.dm = sqrt(sq(x2 - xm) + sq(y2 + ym));
        s.r12 = 1.0 / (dM - s.dm);
    }
    if (s.c1) {
        auto fac = [&](double x, double y, double rp, double& ro, double& p, double& h) {
            ro = (sq(x) + sq(y)) / dis2;
            p = rp / pdis;
            h = sqrt(sqrt(ro));  // (|c| / |f|)^H_pow
        };
        fac(xm, ym, b.rp[M], s.kro, s.kp, s.kh);
        fac(xs, ys, b.rp[So], s.kroS, s.kpS, s.khS);
        if (Sd >= 0) {
            fac(xd, yd, b.rp[Sd], s.kroD, s.kpD, s.khD);
        } else {  // the mirrored centre has the radius of M itself
            s.kroD = s.kro;
            s.kpD = s.kp;
            s.khD = s.kh;
        }
        double c1, s1;
        polar_cs(xm, ym, c1, s1);
        s.C = c1 * cf + s1 * sf;
        s.Sn = c1 * sf - s1 * cf;
    }
    return s;
}

// Fluid f at a Usualy face seen from s.M (state Ms; So's state Ss): Get_par_TVD
// (Gran.cpp:296-472), or in C_1 cells the radial scaling of Setka.cpp:8337-8349
// with Get_par_TVD_radial (Gran.cpp:562-675) for ro and p of the plasma and H1.
template <int GROUP>
__device__ __forceinline__ St5 k5_recon(const K5Rows& rows, const K5Side& s, double r23, bool tracked, int f,
                                        const St5& Ms, const St5& Ss, int* status) {
    St5 o = Ms;
    const double x2 = -s.dM;
    if (s.c1) {
        if (f > 1) return o;
        o.u = Ms.u * s.C - Ms.v * s.Sn;
        o.v = Ms.u * s.Sn + Ms.v * s.C;
        if (f == 0) o.Q = Ms.Q * s.kro;
        if (s.Sd < 0 && !s.axis) return o;
        const St5 p1 = s.Sd >= 0 ? rows.load(f, s.Sd) : Ms;
        if (f == 0) {
            o.ro = linear3r(p1.ro * s.kroD, Ms.ro * s.kro, Ss.ro * s.kroS, s.r12, r23, x2);
            o.p = linear3r(p1.p * s.kpD, Ms.p * s.kp, Ss.p * s.kpS, s.r12, r23, x2);
        } else {
            o.ro = linear3r(p1.ro * s.khD, Ms.ro * s.kh, Ss.ro * s.khS, s.r12, r23, x2);
            o.p = linear3r(p1.p, Ms.p, Ss.p, s.r12, r23, x2);
        }
        return o;
    }
    if (s.Sd < 0) {
        if (s.axis) o.v = linear3r(-Ms.v, Ms.v, Ss.v, s.r12, r23, x2);  // Gran.cpp:308-338
        return o;
    }
    const St5 p1 = rows.load(f, s.Sd);
    if (GROUP == kAnyGroup && tracked) {  // Gran.cpp:345-426
        const double r = s.r12;
        o.ro = (p1.ro - Ms.ro) * r * (0.0 - x2) + Ms.ro;
        o.p = (p1.p - Ms.p) * r * (0.0 - x2) + Ms.p;
        o.u = (p1.u - Ms.u) * r * (0.0 - x2) + Ms.u;
        o.v = (p1.v - Ms.v) * r * (0.0 - x2) + Ms.v;
        o.Q = (p1.Q - Ms.Q) * r * (0.0 - x2) + Ms.Q;
        if (o.ro <= 0.0) o.ro = Ms.ro;
        if (o.p <= 0.0) o.p = Ms.p;
        return o;
    }
    o.ro = linear3r(p1.ro, Ms.ro, Ss.ro, s.r12, r23, x2);
    o.p = linear3r(p1.p, Ms.p, Ss.p, s.r12, r23, x2);
    o.u = linear3r(p1.u, Ms.u, Ss.u, s.r12, r23, x2);
    o.v = linear3r(p1.v, Ms.v, Ss.v, s.r12, r23, x2);
    if (f == 0) {
        o.Q = linear3r(p1.Q, Ms.Q, Ss.Q, s.r12, r23, x2);
        if (o.ro <= 0.0 || o.p <= 0.0) *status |= ST_TVD_BAD;  // the reference exits (Gran.cpp:444-455)
    }
    return o;
}

// The two states of fluid f at a boundary face of cell `own` (Gran.cpp:205-289
// and 486-545, Setka.cpp:8392-8440).
__device__ __forceinline__ void k5_boundary(const gelios_params& P, const K5Rows& rows, const K5Side& s, int ft,
                                            double x2, double y2, int f, const St5& own, St5& L, St5& R) {
    L = own;
    R = own;
    if (ft == G_EXTERN) {
        if (f == 0 && R.u >= 0.0) R.u = P.extern_u_par;
    } else if (ft == G_INNER_SPHERE) {
        // plasma and H1 of the solar wind, H2..H4 of the cell
        if (f == 0) {
            L.ro = own.ro * s.kro;
            L.Q = own.Q * s.kro;
            L.p = own.p * s.kp;
            R = inner_sphere_state(P, x2, y2);
        } else if (f == 1) {
            L.ro = own.ro * s.kh;
            const double dist = sqrt(x2 * x2 + y2 * y2);
            R.ro = 0.0000001;
            R.p = (0.0000001 * P.chi * P.chi / (P.gamma * 14.1344 * 14.1344));
            R.u = P.chi * x2 / dist;
            R.v = P.chi * y2 / dist;
        }
    } else if (ft == G_INPUT) {
        // plasma and H4 of the LISM, H1..H3 of the cell
        if (f == 0) {
            R = input_state(P);
        } else if (f == 4) {
            R.ro = 1.0;
            R.p = 0.5;
            R.u = P.in_u;  // Velosity_inf
            R.v = 0.0;
        }
    } else if (ft == G_AXIS) {
        if (s.c1) {
            if (f == 0) {
                L.ro = own.ro * s.kro;
                L.Q = own.Q * s.kro;
                L.p = own.p * s.kp;
            } else if (f == 1) {
                L.ro = own.ro * s.kh;
            }
            if (f <= 1) {
                L.u = own.u * s.C - own.v * s.Sn;
                L.v = own.u * s.Sn + own.v * s.C;
            }
        } else if (s.Sd >= 0) {  // Gran.cpp:486-519
            const St5 p1 = rows.load(f, s.Sd);
            L.v = linear3r(p1.v, own.v, -own.v, s.r12, -0.5 / s.dM, -s.dM);
        }
        R = L;
        R.v = -R.v;
    }
}

// Go_5_komponent face units (the face loop of Setka.cpp:8300-8570): each face
// once, after the motion.  The geometry of both sides' reconstructions once,
// then fluid by fluid: both sides' states, the HLLC flux through the moving
// face (on tracked faces the plasma takes the exact Godunov flux and HLLC's
// tracer flux), F*S into the unit's row (the reference evaluates the face
// from each side; the two results are negatives of each other up to
// rounding).  Flux rows: plasma mass, mom x, mom y, energy, Q (0-4), then
// mass, mom x, mom y, energy of H1..H4 (5-20).  Returns the minimum of the
// CFL candidates of each updated side, H1's only where that side is not
// C_centr (Setka.cpp:8500): kurant * distance / the largest wave speed.
// Holding all 21 fields of four cells at once took 255 registers and spilled,
// in one launch of every kind of unit: 223 us on the 200k grid (401k units,
// ncu).  One fluid at a time in a launch per group: 73 us for the plain units
// at 96 registers (21, 30, 19 us for the C_1, tracked and one-sided ones
// beside them, 35 for the tracked before a lane took a fluid); 80 or 128 registers, or the fluids unrolled: 1-5% slower per
// step.  Bound by the latency of its loads and FP64 chains.
// COOP: a warp evaluates one tracked unit, a lane per fluid.
template <int GROUP, bool COOP>
__device__ __forceinline__ double k5_face_body(const DevMesh& d, const gelios_params& P, const StepBuffers& b,
                                               const double* __restrict__ hcur, double* __restrict__ fl, int u,
                                               int& status) {
    // a face whose two end points lie on one surface counts as tracked even on
    // the grid's boundary, so the tracked units are not all interior ones
    constexpr bool USUALY = GROUP != kAnyGroup;
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    const size_t nu = d.n_units;
    const int K = d.u_cell[u], nb = d.u_nb[u];
    const uint32_t info = d.u_info[u];
    const uint32_t cf = (info >> UI_CF_OWN) & 15u, nbf = (info >> UI_CF_NB) & 15u;
    const double x = b.cx[K], y = b.cy[K];
    const bool procK = !(sq(x) + sq(y) < d.r11_sq);
    double x3 = 0.0, y3 = 0.0;
    bool procN = false;
    if (nb >= 0) {
        x3 = b.cx[nb];
        y3 = b.cy[nb];
        procN = !(sq(x3) + sq(y3) < d.r11_sq);
    }
    if (!(procK || procN)) return inf;
    const int ft = USUALY ? static_cast<int>(G_USUALY) : static_cast<int>(info & SI_TYPE_MASK);
    const bool tracked = COOP;
    const int A = d.u_A[u], B = d.u_B[u];
    const double xa = d.X[A], ya = d.Y[A], xb = d.X[B], yb = d.Y[B];
    const double x2 = (xa + xb) / 2.0, y2 = (ya + yb) / 2.0;
    const double x4 = (d.X2[A] + d.X2[B]) / 2.0, y4 = (d.Y2[A] + d.Y2[B]) / 2.0;
    const double S = sqrt(sq(xb - xa) + sq(yb - ya)), rS = 1.0 / S;
    const double n1 = (yb - ya) * rS, n2 = -((xb - xa) * rS);
    const double W = ((x4 - x2) * n1 + (y4 - y2) * n2) / *b.dt_cur;
    const double dK = sqrt(sq(x - x2) + sq(y - y2)), dN = sqrt(sq(x3 - x2) + sq(y3 - y2));
    const double dis2 = sq(x2) + sq(y2);
    const bool radial = GROUP != kPlainGroup && ((cf & CF_C1) || ft == G_INNER_SPHERE || (nb >= 0 && (nbf & CF_C1)));
    double pdis = 1.0, cfc = 1.0, sfc = 0.0;
    if (radial) {
        pdis = pow2g(sqrt(dis2), 2.0 * P.gamma);
        polar_cs(x2, y2, cfc, sfc);
    }
    // an inner-sphere face scales its cell as a C_1 side does
    const K5Side sK = k5_side<GROUP>(b, K, x, y, nb >= 0 ? nb : K, nb >= 0 ? x3 : x, nb >= 0 ? y3 : y, d.u_sd[u],
                                     ft == G_INNER_SPHERE ? (cf | CF_C1) : cf, x2, y2, dK, dN, dis2, pdis, cfc, sfc);
    K5Side sN{};
    double r23 = 0.0;
    if (USUALY || ft == G_USUALY) {
        sN = k5_side<GROUP>(b, nb, x3, y3, K, x, y, d.u_sd2[u], nbf, x2, y2, dN, dK, dis2, pdis, cfc, sfc);
        r23 = 1.0 / (-dK - dN);
    }
    const K5Rows rows{b.cur, hcur, static_cast<size_t>(d.n_cells)};
    double um = 0.0, um1 = 0.0;  // largest wave speed without H1, of H1
    // fluid f: the two states, the HLLC flux and its wave speed; the flux row
    auto flux = [&](int f, St5& L, St5& R, double (&F)[5]) {
        const St5 own = rows.load(f, K);
        if (USUALY || ft == G_USUALY) {
            const St5 oth = rows.load(f, nb);
            constexpr int G = COOP ? kAnyGroup : GROUP;
            L = k5_recon<G>(rows, sK, r23, tracked, f, own, oth, &status);
            R = k5_recon<G>(rows, sN, r23, tracked, f, oth, own, &status);
        } else {
            k5_boundary(P, rows, sK, ft, x2, y2, f, own, L, R);
        }
        return hllc_lean<double, true, true>(P.gamma, L, R, W, n1, n2, f == 0 && (info & SI_NP), F);
    };
    auto store = [&](int f, const double* F) {
        double* o = fl + (f == 0 ? 0 : 1 + 4 * f) * nu + u;
#pragma unroll
        for (int k = 0; k < 4; k++) o[k * nu] = F[k] * S;
        if (f == 0) o[4 * nu] = F[4] * S;
    };
    if constexpr (COOP) {
        // a lane per fluid (the lanes above 4 repeat H4), then the exact
        // solution of the plasma's states by the whole warp
        const unsigned full = 0xffffffffu;
        const int lane = threadIdx.x & 31, f = lane < 4 ? lane : 4;
        St5 L, R;
        double F[5];
        const double UU = flux(f, L, R, F);
        __syncwarp();
        double q1[5] = {L.ro, L.p, L.u, L.v, 0.0}, q2[5] = {R.ro, R.p, R.u, R.v, 0.0};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            q1[k] = __shfl_sync(full, q1[k], 0);
            q2[k] = __shfl_sync(full, q2[k], 0);
        }
        double nv[3] = {n1, n2, 0.0}, qq[5], ds[3];
        um = godunov_dev<true>(P.gamma, P.kurant, q1, q2, nv, qq, ds, W, 1.0, P.godunov_max_iter, &status);
        um = um > 0.0 ? um : 0.0;
        if (f == 0) {
            F[0] = qq[0];
            F[1] = qq[1];
            F[2] = qq[2];
            F[3] = qq[4];
        }
        if (lane < 5) store(f, F);
#pragma unroll
        for (int j = 0; j < 5; j++) {
            const double w = __shfl_sync(full, UU, j);
            if (j == 1) um1 = w > um1 ? w : um1;
            else um = w > um ? w : um;
        }
    } else {
#pragma unroll 1
        for (int f = 0; f < 5; f++) {
            St5 L, R;
            double F[5];
            const double UU = flux(f, L, R, F);
            store(f, F);
            if (f == 1) um1 = UU > um1 ? UU : um1;
            else um = UU > um ? UU : um;
        }
    }
    const double ua = um1 > um ? um1 : um;
    double t = inf;
    if (procK) t = dmin_ref(t, P.kurant * dK / ((cf & CF_CENTR) ? um : ua));
    if (nb >= 0 && procN) t = dmin_ref(t, P.kurant * dN / ((nbf & CF_CENTR) ? um : ua));
    return t;
}
template <int GROUP, int MINB>
__global__ void __launch_bounds__(128, MINB) k5_face_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                            const double* __restrict__ hcur, double* __restrict__ fl,
                                                            int n_launch) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double t = __longlong_as_double(0x7ff0000000000000LL);
    int status = 0;
    if (i < n_launch) {
        const int u = GROUP == kPlainGroup ? i : GROUP == kC1Group ? d.u_c1 + i : d.u_tr1 + i;
        t = k5_face_body<GROUP, false>(d, P, b, hcur, fl, u, status);
    }
    block_reduce_commit(t, 0, 0, status, b.dt_acc, b.counters, b.status);
}
// The tracked units, one warp each: the five fluids in five lanes, then the
// exact solver's bisection warp-cooperatively (one thread per unit holds up
// its block for 30 iterations in a row).  With the fluids one after another in
// every lane the 1150 units of the 200k grid took as many issue slots of the
// FP64 pipes, which the face kernels share, as a fifth of the 328k plain ones.
// 20 steps of that grid: 5870 -> 5603 us.
__global__ void __launch_bounds__(64) k5_tracked_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                        const double* __restrict__ hcur, double* __restrict__ fl) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    double t = __longlong_as_double(0x7ff0000000000000LL);
    int status = 0;
    if (i < d.u_tr1 - d.u_tr0) t = k5_face_body<kAnyGroup, true>(d, P, b, hcur, fl, d.u_tr0 + i, status);
    block_reduce_commit(t, 0, 0, status, b.dt_acc, b.counters, b.status);
}

// conservative update of one hydrogen fluid with its sources and the
// cylindrical terms (Setka.cpp:8808-8940)
__device__ __forceinline__ void k5_update_h(double ga, const double* pot, double ro_H, double p_H, double u_H,
                                            double v_H, double q1, double q21, double q22, double q3, double VV,
                                            double rV2, double ry, double dt, double ro_floor, double p_floor,
                                            double* out, int& nro, int& npc) {
    const double gm1 = ga - 1, rg1 = 1.0 / gm1, vy = v_H * ry, ek = ro_H * (u_H * u_H + v_H * v_H) * 0.5;
    double ro3 = ro_H * VV - dt * (pot[0] * rV2 + ro_H * vy - q1);
    if (ro3 <= 0) {
        ro3 = ro_floor;
        nro++;
    }
    const double rro3 = 1.0 / ro3;
    const double u3 = (ro_H * u_H * VV - dt * (pot[1] * rV2 + ro_H * vy * u_H - q21)) * rro3;
    const double v3 = (ro_H * v_H * VV - dt * (pot[2] * rV2 + ro_H * vy * v_H - q22)) * rro3;
    double p3 = (((p_H * rg1 + ek) * VV - dt * (pot[3] * rV2 + vy * (ga * p_H * rg1 + ek) - q3)) -
                 0.5 * ro3 * (u3 * u3 + v3 * v3)) *
                gm1;
    if (p3 <= 0) {
        p3 = p_floor;
        npc++;
    }
    out[0] = ro3;
    out[1] = p3;
    out[2] = u3;
    out[3] = v3;
}

// Go_5_komponent cell update (Setka.cpp:8570-8950) from the face units' fluxes
// summed in Grans order: multi-fluid charge exchange, cylindrical 1/y terms,
// clamps; it also refills the geometry cache for the next step.  The area
// before the motion comes from that cache; a quadrilateral's corners come in
// one load.
// 32 cells per warp in three phases, every lane busy in each: one lane per
// cell (geometry, the plasma's state, into shared memory), four rounds of
// eight cells x four hydrogen fluids (a fluid's exchange rate, its update;
// the rates summed over the cell's four lanes in fluid order), one lane per
// cell again (the plasma's update).  With one thread per cell throughout, 21
// fields and 21 flux sums took 128 registers: 89 us against 78 on the 200k
// grid (97 before the flux rows were the units'; ncu).
__global__ void __launch_bounds__(128, 6) k5_update_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                           const double* __restrict__ fl,
                                                           const double* __restrict__ hcur, double* __restrict__ hnxt) {
    // per-cell values of the block's 128 cells: u, v, ro, p/ro, V/V2, 1/V2, 1/y, then the summed exchange terms
    __shared__ double sd[10][128];
    __shared__ int si[128];    // kind of the cell (Cell_type), -1: not updated
    __shared__ int4 ssu[128];  // the units of a quadrilateral's four slots (s_unit), x < 0: another cell
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wbase = threadIdx.x & ~31, th_ = threadIdx.x;
    const int c0 = blockIdx.x * blockDim.x + wbase, c = c0 + lane;
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    double tmin = inf;
    int nro = 0, npc = 0;
    const size_t nc = d.n_cells, nu = d.n_units;
    const K5Rows rows{b.cur, hcur, nc};
    const double ga = P.gamma, gm1 = ga - 1, rg1 = 1.0 / gm1, dt = *b.dt_cur;
    St5 pl{};
    int kind = -1;
    if (c < d.n_cells) {
        const uint32_t cfl = d.cflags[c];
        const double x = b.cx[c], y = b.cy[c];
        const bool proc = !(sq(x) + sq(y) < d.r11_sq);
        {
            const int g0 = d.gstart[c];
            int4 su = make_int4(-1, -1, -1, -1);
            if (d.gstart[c + 1] - g0 == 4)
                su = make_int4(d.s_unit[g0], d.s_unit[g0 + 1], d.s_unit[g0 + 2], d.s_unit[g0 + 3]);
            ssu[th_] = su;
        }
        double Volume2 = 0.0;
        {  // the next step's geometry cache from the moved points (see mk2_update_cell)
            double xn, yn, vs, vol;
            const int4 qc = d.qcorner[c];
            if (qc.x >= 0) {
                const double qx[4] = {d.X2[qc.x], d.X2[qc.y], d.X2[qc.z], d.X2[qc.w]};
                const double qy[4] = {d.Y2[qc.x], d.Y2[qc.y], d.Y2[qc.z], d.Y2[qc.w]};
                quad_geometry(qx, qy, xn, yn, vs, vol);
                Volume2 = vs;
            } else {
                const int s0 = d.cstart[c], n = d.cstart[c + 1] - s0, g0 = d.gstart[c], g1 = d.gstart[c + 1];
                const int32_t* con = d.contour + s0;
                centroid(con, n, d.X2, d.Y2, xn, yn);
                vs = area(con, n, d.sA, d.sB, g0, g1, d.X2, d.Y2, false);
                vol = volume_rotate(con, n, d.X2, d.Y2);
                if (proc) Volume2 = area(con, n, d.sA, d.sB, g0, g1, d.X2, d.Y2, true);
            }
            b.cx_next[c] = xn;
            b.cy_next[c] = yn;
            if (cfl & CF_RP) b.rp_next[c] = pow2g(sqrt(sq(xn) + sq(yn)), 2 * P.gamma);
            if (!(cfl & CF_CENTR)) {
                b.vs_next[c] = vs;
                b.vol_next[c] = vol;
            }
        }
        if (proc) {
            tmin = 10000000.0;  // `time` starts at 1e7 in every step (Setka.cpp:8286)
            kind = d.ctype[c];
            double Volume;
            if (!(cfl & CF_CENTR)) {
                Volume = b.vs[c];
            } else {  // the cache holds no area of the C_centr cells
                const int s0 = d.cstart[c];
                Volume = area(d.contour + s0, d.cstart[c + 1] - s0, d.sA, d.sB, d.gstart[c], d.gstart[c + 1], d.X, d.Y,
                              false);
            }
            pl = rows.load(0, c);
            const double rV2 = 1.0 / Volume2;
            sd[0][th_] = pl.u;
            sd[1][th_] = pl.v;
            sd[2][th_] = pl.ro;
            sd[3][th_] = pl.p / pl.ro;
            sd[4][th_] = Volume * rV2;
            sd[5][th_] = rV2;
            sd[6][th_] = 1.0 / y;
        }
    }
    si[th_] = kind;
    __syncwarp();
    // the flux rows first .. first + N - 1 of cell k's faces, summed in Grans order
    auto sums = [&](int k, int t, int first, double* out, auto n_const) {
        constexpr int N = decltype(n_const)::value;
#pragma unroll
        for (int q = 0; q < N; q++) out[q] = 0.0;
        const double* r = fl + first * nu;
        const int4 s4 = ssu[t];
        if (s4.x >= 0) {  // quadrilaterals: all loads in flight together
            const int su[4] = {s4.x, s4.y, s4.z, s4.w};
            double a[N][4];
#pragma unroll
            for (int q = 0; q < N; q++)
#pragma unroll
                for (int j = 0; j < 4; j++) a[q][j] = r[q * nu + (su[j] >> 1)];
#pragma unroll
            for (int q = 0; q < N; q++)
#pragma unroll
                for (int j = 0; j < 4; j++) out[q] = out[q] + ((su[j] & 1) ? -a[q][j] : a[q][j]);
        } else {
            const int g0 = d.gstart[k], nf = d.gstart[k + 1] - g0;
            for (int j = 0; j < nf; j++) {
                const int w = d.s_unit[g0 + j];
#pragma unroll
                for (int q = 0; q < N; q++) {
                    const double v = r[q * nu + (w >> 1)];
                    out[q] = out[q] + ((w & 1) ? -v : v);
                }
            }
        }
    };
    const int f = lane & 3, q0 = lane & ~3;
#pragma unroll 1
    for (int rd = 0; rd < 4; rd++) {
        const int t = wbase + 8 * rd + (lane >> 2), k = c0 + 8 * rd + (lane >> 2);
        const int kt = si[t];
        St5 h{1.0, 1.0, 0.0, 0.0, 0.0};
        double u = 0.0, v = 0.0, nu4 = 0.0, uhm = 0.0, th = 0.0, mu = 0.0, mv = 0.0, mt = 0.0, s2 = 0.0;
        double PH[4];
        if (kt >= 0) {  // charge exchange with the plasma (Setka.cpp:8575-8660)
            u = sd[0][t];
            v = sd[1][t];
            const double ro = sd[2][t], pro = sd[3][t];
            h = rows.load(f + 1, k);
            sums(k, t, 5 + 4 * f, PH, std::integral_constant<int, 4>{});
            th = 2.0 * h.p / h.ro;
            const double du2 = sq(u - h.u) + sq(v - h.v), a = pro + th;
            const double UM2 = du2 + (64.0 / (9.0 * kPi)) * a, UH2 = du2 + (4.0 / kPi) * a;
            const double r = rsqrt(UM2);
            uhm = sqrt(UH2) * r;
            nu4 = ro * h.ro * (UM2 * r) * sq(1.0 - P.a_2 * (0.5 * log(UM2)));
            mu = nu4 * (h.u - u);
            mv = nu4 * (h.v - v);
            mt = nu4 * ((sq(h.u) + sq(h.v) - sq(u) - sq(v)) / 2.0 + uhm * (th - pro));
            s2 = nu4 * ((sq(u) + sq(v)) / 2.0 + uhm * pro);
        }
        double S1 = 0.0, S2 = 0.0, Mu = 0.0, Mv = 0.0, MT = 0.0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            S1 += __shfl_sync(full, nu4, q0 + j);
            S2 += __shfl_sync(full, s2, q0 + j);
            Mu += __shfl_sync(full, mu, q0 + j);
            Mv += __shfl_sync(full, mv, q0 + j);
            MT += __shfl_sync(full, mt, q0 + j);
        }
        if (kt >= 0) {
            if (f == 0) {
                sd[7][t] = Mu;
                sd[8][t] = Mv;
                sd[9][t] = MT;
            }
            // hydrogen sources by cell kind (Setka.cpp:8734-8806)
            const int born = (kt == C_1 || kt == C_CENTR) ? 0 : (kt == C_2 || kt == C_3) ? 1 : kt == C_4 ? 2 : 3;
            double out[4] = {h.ro, h.p, h.u, h.v};
            if (!(f == 0 && kt == C_CENTR)) {
                const double kk = f == born ? 1.0 : 0.0;
                const double q1h = kNHOverKn * (kk * S1 - nu4);
                const double q21h = kNHOverKn * (kk * S1 * u - nu4 * h.u);
                const double q22h = kNHOverKn * (kk * S1 * v - nu4 * h.v);
                const double q3h = kNHOverKn * (kk * S2 - nu4 * ((sq(h.u) + sq(h.v)) / 2.0 + uhm * th));
                // floors: Setka.cpp:8817, 8829, 8859, 8871, 8893, 8905, 8927, 8939
                const double rf = f == 0 ? 0.0000001 : 0.000001;
                const double pf = f == 3 ? 0.0000001 : 0.000001;
                k5_update_h(ga, PH, h.ro, h.p, h.u, h.v, q1h, q21h, q22h, q3h, sd[4][t], sd[5][t], sd[6][t], dt, rf, pf,
                            out, nro, npc);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) hnxt[(4 * f + j) * nc + k] = out[j];
        }
    }
    __syncwarp();
    if (kind >= 0) {
        const double ro = pl.ro, u = pl.u, v = pl.v, p = pl.p, Q = pl.Q;
        St5 o = pl;
        if (kind != C_CENTR) {
            const double cp = P.src_coef;  // n_p_LISM_ / Kn_
            const double q2_1 = cp * sd[7][th_], q2_2 = cp * sd[8][th_], q3 = cp * sd[9][th_];
            const double VV = sd[4][th_], rV2 = sd[5][th_], vy = v * sd[6][th_];
            double Pt[5];
            sums(c, th_, 0, Pt, std::integral_constant<int, 5>{});
            o.ro = ro * VV - dt * (Pt[0] * rV2 + ro * vy);
            o.Q = Q * VV - (dt * rV2) * Pt[4] - dt * Q * vy;
            if (o.ro <= 0.0) {
                o.ro = P.ro_floor;
                nro++;
            }
            const double rro3 = 1.0 / o.ro, ek = ro * (u * u + v * v) * 0.5;
            o.u = (ro * u * VV - dt * (Pt[1] * rV2 + ro * vy * u - q2_1)) * rro3;
            o.v = (ro * v * VV - dt * (Pt[2] * rV2 + ro * vy * v - q2_2)) * rro3;
            o.p = (((p * rg1 + ek) * VV - dt * (Pt[3] * rV2 + vy * (ga * p * rg1 + ek) - q3)) -
                   0.5 * o.ro * (o.u * o.u + o.v * o.v)) *
                  gm1;
            if (o.p <= 0) {
                o.p = P.p_floor;
                npc++;
            }
        }
        b.nxt[0][c] = o.ro;
        b.nxt[1][c] = o.p;
        b.nxt[2][c] = o.u;
        b.nxt[3][c] = o.v;
        b.nxt[4][c] = o.Q;
    }
    block_reduce_commit(tmin, nro, npc, 0, b.dt_acc, b.counters, b.status);
}

// ------------------------------------------------------------------ MHD + pickup protons
// GELIOS_FORM_MHD_PUI (no reference step).  The ion fluid's gas-dynamic
// rows (ro, p, u, v, Q) are the state rows of the moving-grid step, so
// surface tracking and the rails run on them unchanged; the extra rows hold
// the ion's w (u_phi) and B (x, y, phi) and the pickup protons' ro, p, u, v.
enum : int { kXw = 0, kXbx, kXby, kXbz, kXro, kXp, kXu, kXv, kMhdExtra };
constexpr int kMhdFlux = 13;  // per unit: ion mass, mom x, y, phi, energy, Bx, By, Bphi, Q; pickup mass, mom x, y, energy

struct Ext8 {
    double f[kMhdExtra];
};

__device__ __forceinline__ Ext8 load_ext(const double* __restrict__ hs, size_t nc, int c) {
    Ext8 e;
#pragma unroll
    for (int k = 0; k < kMhdExtra; k++) e.f[k] = hs[k * nc + c];
    return e;
}
// mirror image across the axis: radial and azimuthal components change sign
__device__ __forceinline__ void mirror_ext(Ext8& e) {
    e.f[kXw] = -e.f[kXw];
    e.f[kXby] = -e.f[kXby];
    e.f[kXbz] = -e.f[kXbz];
    e.f[kXv] = -e.f[kXv];
}

// Gran::Get_par's boundary rules (Gran.cpp:205-289) applied to the extra
// rows; `ion` is the ion state the same rule gave (inner sphere: the wind).
__device__ __forceinline__ Ext8 get_par_ext(const gelios_params& P, const gelios_mhd_params& M, int ft,
                                            const Ext8& own, const double* __restrict__ hs, size_t nc, int nb,
                                            double fx, double fy, const St5& ion) {
    Ext8 e = own;
    if (ft == G_USUALY) {
        e = load_ext(hs, nc, nb);
    } else if (ft == G_EXTERN) {
        if (e.f[kXu] >= 0.0) e.f[kXu] = P.extern_u_par;
    } else if (ft == G_AXIS) {
        mirror_ext(e);
    } else if (ft == G_INNER_SPHERE) {
        const double dist = sqrt(fx * fx + fy * fy);
        e.f[kXw] = 0.0;
        e.f[kXbx] = 0.0;
        e.f[kXby] = 0.0;
        e.f[kXbz] = M.inner_bphi * (P.R1 / dist) * (fy / dist);
        e.f[kXro] = M.pui_inner_ro * ion.ro;
        e.f[kXp] = M.pui_inner_p * ion.p;
        e.f[kXu] = ion.u;
        e.f[kXv] = ion.v;
    } else if (ft == G_INPUT) {
        e.f[kXw] = 0.0;
        e.f[kXbx] = M.lism_bx;
        e.f[kXby] = M.lism_by;
        e.f[kXbz] = M.lism_bz;
        e.f[kXro] = M.pui_in_ro;
        e.f[kXp] = M.pui_in_p;
        e.f[kXu] = P.in_u;
        e.f[kXv] = P.in_v;
    }
    return e;
}

// All 13 rows at a Usualy face seen from M (ion Ms, extra Me, centre Mx,My,
// flags mf), with the cell So across the face already loaded (Ss, Se,
// centre Sx,Sy) and Sosed_down Sd: the ion rows follow mk2_usualy_side
// (Get_par_TVD / Get_par_TVD_radial in C_1 cells), the extra rows tvd_ext's
// rule, with the stencil distances computed once for both.
__device__ __forceinline__ void mhd_usualy_side(const double* const* st, const double* __restrict__ hs, size_t nc,
                                                const double* cx, const double* cy, const double* rp, double fx,
                                                double fy, double dis, double pdis, const St5& Ms, const Ext8& Me,
                                                double Mx, double My, double rpM, uint32_t mf, int So, const St5& Ss,
                                                const Ext8& Se, double Sx, double Sy, int Sd, bool tracked,
                                                double rM, double rS, double dM, double dS, St5& oi, Ext8& oe,
                                                int* status) {
    // rM, rS: |centroid| of M and So; dM, dS: face centre to those centroids
    if (mf & CF_C1) {
        oi = mk2_usualy_side_d(st, cx, cy, rp, fx, fy, dis, pdis, Ms, Mx, My, rpM, mf, So, Sd, tracked, rM, rS, dM,
                               dS, status);
        oe = Me;
        return;
    }
    oi = Ms;
    oe = Me;
    if (Sd < 0) {
        if (mf & CF_AXIS) {  // Gran.cpp:308-338
            const double dist2 = dM;
            const double dist3 = dS;
            const double dist1 = sqrt(sq(fx - Mx) + sq(fy - (-My)));
            oi.v = linear3(-dist1, -Ms.v, -dist2, Ms.v, dist3, Ss.v, 0.0);
        }
        return;
    }
    const St5 s1 = load_state(st, Sd);
    const Ext8 e1 = load_ext(hs, nc, Sd);
    const double dist2 = dM;
    const double dist1 = sqrt(sq(fx - cx[Sd]) + sq(fy - cy[Sd]));
    const double r12 = 1.0 / (-dist1 - (-dist2)), x2 = -dist2;
    if (tracked) {  // Gran.cpp:345-426
        oi.ro = (s1.ro - Ms.ro) * r12 * (0.0 - x2) + Ms.ro;
        oi.p = (s1.p - Ms.p) * r12 * (0.0 - x2) + Ms.p;
        oi.u = (s1.u - Ms.u) * r12 * (0.0 - x2) + Ms.u;
        oi.v = (s1.v - Ms.v) * r12 * (0.0 - x2) + Ms.v;
        oi.Q = (s1.Q - Ms.Q) * r12 * (0.0 - x2) + Ms.Q;
        if (oi.ro <= 0.0) oi.ro = Ms.ro;
        if (oi.p <= 0.0) oi.p = Ms.p;
#pragma unroll
        for (int k = 0; k < kMhdExtra; k++) oe.f[k] = (e1.f[k] - Me.f[k]) * r12 * (0.0 - x2) + Me.f[k];
    } else {
        const double dist3 = dS;
        const double r23 = 1.0 / (-dist2 - dist3);
        oi.ro = linear3r(s1.ro, Ms.ro, Ss.ro, r12, r23, x2);
        oi.p = linear3r(s1.p, Ms.p, Ss.p, r12, r23, x2);
        oi.u = linear3r(s1.u, Ms.u, Ss.u, r12, r23, x2);
        oi.v = linear3r(s1.v, Ms.v, Ss.v, r12, r23, x2);
        oi.Q = linear3r(s1.Q, Ms.Q, Ss.Q, r12, r23, x2);
        if (oi.ro <= 0.0 || oi.p <= 0.0) *status |= ST_TVD_BAD;  // the reference exits (Gran.cpp:444-455)
#pragma unroll
        for (int k = 0; k < kMhdExtra; k++) oe.f[k] = linear3r(e1.f[k], Me.f[k], Se.f[k], r12, r23, x2);
    }
    if (!(oe.f[kXro] > 0.0)) oe.f[kXro] = Me.f[kXro];
    if (!(oe.f[kXp] > 0.0)) oe.f[kXp] = Me.f[kXp];
}

// Ion MHD flux through a face with unit normal (n1, n2) moving with normal
// speed W: both states go to the face frame (normal n, tangent t = (-n2,
// n1), phi), Solvers::HLLDQ_Korolkov's HLLD (metod 3) solves along the
// frame's x axis with its fan sampled at W (hlldq_impl<true>: F - W U of
// the region containing W, as HLLC_2d_Korolkov_b_s does for moving faces),
// and the momentum and field fluxes go back to (x, y).  out: mass, mom x,
// mom y, mom phi, energy, Bx, By, Bphi, Q.  Returns 1 / max(|SL|, |SR|).
template <typename TF>
__device__ __forceinline__ double mhd_face_flux(double ga, const St5& iL, const Ext8& eL, const St5& iR,
                                                const Ext8& eR, double n1, double n2, double W, double* out) {
    const double t1 = -n2, t2 = n1;
    double L[9], R[9];
    L[0] = iL.ro;
    L[1] = iL.Q;
    L[2] = iL.p;
    L[3] = iL.u * n1 + iL.v * n2;
    L[4] = iL.u * t1 + iL.v * t2;
    L[5] = eL.f[kXw];
    L[6] = eL.f[kXbx] * n1 + eL.f[kXby] * n2;
    L[7] = eL.f[kXbx] * t1 + eL.f[kXby] * t2;
    L[8] = eL.f[kXbz];
    R[0] = iR.ro;
    R[1] = iR.Q;
    R[2] = iR.p;
    R[3] = iR.u * n1 + iR.v * n2;
    R[4] = iR.u * t1 + iR.v * t2;
    R[5] = eR.f[kXw];
    R[6] = eR.f[kXbx] * n1 + eR.f[kXby] * n2;
    R[7] = eR.f[kXbx] * t1 + eR.f[kXby] * t2;
    R[8] = eR.f[kXbz];
    double F[8], FQ;
    const double tinv = hlld_face_moving<TF>(ga, L, R, W, F, &FQ);
    out[0] = F[0];
    out[1] = n1 * F[1] + t1 * F[2];
    out[2] = n2 * F[1] + t2 * F[2];
    out[3] = F[3];
    out[4] = F[7];
    out[5] = n1 * F[4] + t1 * F[5];
    out[6] = n2 * F[4] + t2 * F[5];
    out[7] = F[6];
    out[8] = FQ;
    return tinv;
}

// One face unit of the MHD form, after the motion: reconstructions of both
// sides (ion rows: the moving-grid rules of Setka.cpp:10204-10276, extra
// rows: mhd_usualy_side / get_par_ext) on the pre-motion points, face speed
// from the moved points, HLLD for the ions and HLLC for the pickup protons,
// 13 flux rows times S into the unit's rows,
// CFL candidates of both fluids.  BLOCK x MINB: the launch shape (threads
// per block, minimum resident blocks per SM, which caps the registers).
// PLAIN: a unit of the plain interior group [0, u_c1) (see mk2_recon_unit).
template <typename TF, bool PLAIN = false>
__device__ __forceinline__ double mhd_face_body(const DevMesh& d, const gelios_params& P, const gelios_mhd_params& M,
                                                const StepBuffers& b, const double* __restrict__ hs,
                                                double* __restrict__ fl, int u, int& status) {
    double tmin_u = __longlong_as_double(0x7ff0000000000000LL);
    {
        const size_t nc = d.n_cells, nu = d.n_units;
        const int K = d.u_cell[u], nb = d.u_nb[u];
        const uint32_t info = d.u_info[u];
        const double x = b.cx[K], y = b.cy[K];
        // as mk2_recon_unit: the R11 test without a square root, the radii
        // only where a radial reconstruction reads them, the distances once
        const double aK = sq(x) + sq(y);
        const bool procK = !(aK < d.r11_sq);
        double x3 = 0.0, y3 = 0.0, aN = 0.0;
        bool procN = false;
        if (nb >= 0) {
            x3 = b.cx[nb];
            y3 = b.cy[nb];
            aN = sq(x3) + sq(y3);
            procN = !(aN < d.r11_sq);
        }
        if (procK || procN) {
            const double rK = PLAIN ? 0.0 : sqrt(aK), rN = PLAIN ? 0.0 : sqrt(aN);
            const int A = d.u_A[u], B = d.u_B[u];
            const double xa = d.X[A], ya = d.Y[A], xb = d.X[B], yb = d.Y[B];
            const double x2 = (xa + xb) / 2.0, y2 = (ya + yb) / 2.0;
            const double dK = sqrt(sq(x - x2) + sq(y - y2));
            const double dN = sqrt(sq(x3 - x2) + sq(y3 - y2));
            double t1 = xb - xa, t2 = yb - ya;
            const double nn = sqrt(sq(t1) + sq(t2));
            t1 = t1 / nn;
            t2 = t2 / nn;
            const double n1 = t2, n2 = -t1;
            const double S = nn * (ya + yb) * 0.5;
            const double x4 = (d.X2[A] + d.X2[B]) / 2.0, y4 = (d.Y2[A] + d.Y2[B]) / 2.0;
            const double dt = *b.dt_cur;
            const double W = ((x4 - x2) * n1 + (y4 - y2) * n2) / dt;
            const int ft = PLAIN ? static_cast<int>(G_USUALY) : static_cast<int>(info & SI_TYPE_MASK);
            const uint32_t cmask = PLAIN ? (15u & ~CF_C1) : 15u;
            const uint32_t cf = (info >> UI_CF_OWN) & cmask, nbf = (info >> UI_CF_NB) & cmask;
            const double g2 = 2 * P.gamma;
            const St5 par1 = load_state(b.cur, K);
            const Ext8 ex1 = load_ext(hs, nc, K);
            St5 par11 = par1, par2 = get_par(P, ft, par1, b.cur, nb, x2, y2);
            Ext8 e11 = ex1, e2 = get_par_ext(P, M, ft, ex1, hs, nc, nb, x2, y2, par2);
            const double dis = sqrt(sq(x2) + sq(y2));
            const bool tracked = !PLAIN && (info & SI_GOD) != 0;
            const bool radial = ((cf & CF_C1) && (ft == G_USUALY || ft == G_AXIS)) || ft == G_INNER_SPHERE ||
                                (ft == G_USUALY && (nbf & CF_C1));
            const double pdis = radial ? pow2g(dis, g2) : 1.0;
            if (ft == G_USUALY) {
                const St5 sN = par2;
                const Ext8 eN = e2;
                mhd_usualy_side(b.cur, hs, nc, b.cx, b.cy, b.rp, x2, y2, dis, pdis, par1, ex1, x, y, b.rp[K], cf, nb,
                                sN, eN, x3, y3, d.u_sd[u], tracked, rK, rN, dK, dN, par11, e11, &status);
                mhd_usualy_side(b.cur, hs, nc, b.cx, b.cy, b.rp, x2, y2, dis, pdis, sN, eN, x3, y3, b.rp[nb], nbf, K,
                                par1, ex1, x, y, d.u_sd2[u], tracked, rN, rK, dN, dK, par2, e2, &status);
            } else if (ft == G_INNER_SPHERE) {
                const double radius = rK;
                par11.ro = par11.ro * sq(radius) / sq(dis);
                par11.Q = par11.Q * sq(radius) / sq(dis);
                par11.p = par11.p * (b.rp[K] / pdis);
            } else if (ft == G_AXIS) {
                if (cf & CF_C1) {
                    const double radius = sqrt(sq(x) + sq(y));
                    par11.ro = par11.ro * sq(radius) / sq(dis);
                    par11.Q = par11.Q * sq(radius) / sq(dis);
                    par11.p = par11.p * (b.rp[K] / pdis);
                    polar_perenos(x, y, x2, y2, par11.u, par11.v);
                } else {
                    par11 = tvd_axis(b.cur, b.cx, b.cy, x2, y2, par1, x, y, d.u_sd[u]);
                }
                par2 = par11;
                par2.v = -par2.v;
            }
            double F[kMhdFlux];
            const double tI = mhd_face_flux<TF>(P.gamma, par11, e11, par2, e2, n1, n2, W, F);
            St5 pL, pR;
            pL.ro = e11.f[kXro];
            pL.p = e11.f[kXp];
            pL.u = e11.f[kXu];
            pL.v = e11.f[kXv];
            pL.Q = 0.0;
            pR.ro = e2.f[kXro];
            pR.p = e2.f[kXp];
            pR.u = e2.f[kXu];
            pR.v = e2.f[kXv];
            pR.Q = 0.0;
            FluxOut<double> G;
            const double UUp = hllc_flux<TF>(P.gamma, P.kurant, pL, pR, W, n1, n2, 1.0, 1, false, G);
            F[9] = G.P0;
            F[10] = G.P1;
            F[11] = G.P2;
            F[12] = G.P3;
#pragma unroll
            for (int k = 0; k < kMhdFlux; k++) fl[k * nu + u] = F[k] * S;
            if (procK) {
                const double dist = dK;
                tmin_u = dmin_ref(tmin_u, P.kurant * dist * tI);
                tmin_u = dmin_ref(tmin_u, P.kurant * dist / UUp);
            }
            if (procN) {
                const double distn = dN;
                tmin_u = dmin_ref(tmin_u, P.kurant * distn * tI);
                tmin_u = dmin_ref(tmin_u, P.kurant * distn / UUp);
            }
        }
    }
    return tmin_u;
}

// PLAIN: the plain interior group [0, u_c1) (lean instance); otherwise the
// units [u_c1, n_units).
template <typename TF, int BLOCK, int MINB, bool PLAIN>
__global__ void __launch_bounds__(BLOCK, MINB) mhd_face_kernel(DevMesh d, gelios_params P, gelios_mhd_params M,
                                                               StepBuffers b, const double* __restrict__ hs,
                                                               double* __restrict__ fl) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int u = PLAIN ? i : d.u_c1 + i;
    double tmin_u = __longlong_as_double(0x7ff0000000000000LL);
    int status = 0;
    if (PLAIN ? u < d.u_c1 : u < d.n_units) tmin_u = mhd_face_body<TF, PLAIN>(d, P, M, b, hs, fl, u, status);
    block_reduce_commit(tmin_u, 0, 0, status, b.dt_acc, b.counters, b.status);
}

// Cell update of the MHD form: the MK2 update (Setka.cpp:10386-10468) for
// both fluids with their axisymmetric terms (area-weighted like the
// reference's p (vs1 + vs2)/2) and the fixed charge-exchange sources of the
// ion momentum and energy; refills the geometry cache like mk2_update_cell.
__device__ __forceinline__ void mhd_update_body(const DevMesh& d, const gelios_params& P, const StepBuffers& b,
                                                const double* __restrict__ fl, const double* __restrict__ src,
                                                const double* __restrict__ hcur, double* __restrict__ hnxt, int c,
                                                double& tmark, int& nro, int& npc) {
    const size_t nu = d.n_units, nc = d.n_cells;
    {
        const uint32_t cfl = d.cflags[c];
        double xn, yn;
        double vs2 = 0.0, Volume2 = 0.0;
        // quadrilaterals: the four moved corners from one int4 load, the
        // operations of centroid / area / volume_rotate in registers
        const int4 qc = d.qcorner ? d.qcorner[c] : make_int4(-1, -1, -1, -1);
        if (qc.x >= 0) {
            const double qx[4] = {d.X2[qc.x], d.X2[qc.y], d.X2[qc.z], d.X2[qc.w]};
            const double qy[4] = {d.Y2[qc.x], d.Y2[qc.y], d.Y2[qc.z], d.Y2[qc.w]};
            double vq, volq;
            quad_geometry(qx, qy, xn, yn, vq, volq);
            if (!(cfl & CF_CENTR)) {
                vs2 = vq;
                Volume2 = volq;
                b.vs_next[c] = vq;
                b.vol_next[c] = volq;
            }
        } else {
            const int s0 = d.cstart[c], n = d.cstart[c + 1] - s0;
            const int32_t* con = d.contour + s0;
            centroid(con, n, d.X2, d.Y2, xn, yn);
            if (!(cfl & CF_CENTR)) {
                vs2 = area(con, n, d.sA, d.sB, d.gstart[c], d.gstart[c + 1], d.X2, d.Y2, true);
                Volume2 = volume_rotate(con, n, d.X2, d.Y2);
                b.vs_next[c] =
                    n == 4 ? vs2 : area(con, n, d.sA, d.sB, d.gstart[c], d.gstart[c + 1], d.X2, d.Y2, false);
                b.vol_next[c] = Volume2;
            }
        }
        b.cx_next[c] = xn;
        b.cy_next[c] = yn;
        if (cfl & CF_RP) b.rp_next[c] = pow2g(sqrt(sq(xn) + sq(yn)), 2 * P.gamma);
        const double x = b.cx[c], y = b.cy[c];
        if (!(sqrt(sq(x) + sq(y)) < P.R11)) {
            tmark = 10000000.0;
            const St5 par1 = load_state(b.cur, c);
            const Ext8 e = load_ext(hcur, nc, c);
            if (!(cfl & CF_CENTR)) {
                const double dt = *b.dt_cur;
                const int g0 = d.gstart[c], g1 = d.gstart[c + 1];
                double Pt[kMhdFlux];
#pragma unroll
                for (int k = 0; k < kMhdFlux; k++) Pt[k] = 0.0;
                if (g1 - g0 == 4) {  // quadrilaterals: all flux loads in flight together
                    int su[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) su[j] = d.s_unit[g0 + j];
#pragma unroll
                    for (int k = 0; k < kMhdFlux; k++) {
                        const double* f = fl + k * nu;
                        const double a0 = unit_flux(f, su[0]), a1 = unit_flux(f, su[1]), a2 = unit_flux(f, su[2]),
                                     a3 = unit_flux(f, su[3]);
                        Pt[k] = (((Pt[k] + a0) + a1) + a2) + a3;
                    }
                } else {
                    for (int g = g0; g < g1; g++) {
                        const int w = d.s_unit[g];
#pragma unroll
                        for (int k = 0; k < kMhdFlux; k++) Pt[k] = Pt[k] + unit_flux(fl + k * nu, w);
                    }
                }
                const double q1 = src[c], q2 = src[nc + c], q3 = src[2 * nc + c];
                const double vs1 = b.vs[c], Volume = b.vol[c];
                const double gm1 = P.gamma - 1;
                const double rV2 = 1.0 / Volume2, VV = Volume * rV2;
                const double Am = 0.5 * (vs1 + vs2);
                const double i4p = 1.0 / (4.0 * kPi), i8p = 1.0 / (8.0 * kPi);
                // ions
                const double ro = par1.ro, p = par1.p, u = par1.u, v = par1.v, Q = par1.Q;
                const double w = e.f[kXw], bx = e.f[kXbx], by = e.f[kXby], bz = e.f[kXbz];
                const double bb = bx * bx + by * by + bz * bz;
                const double Sy = p + bb * i8p + ro * w * w - bz * bz * i4p;
                const double Sphi = -(ro * v * w - by * bz * i4p);
                const double Sbz = v * bz - w * by;
                double ro3 = ro * VV - dt * (Pt[0] * rV2);
                const double Q3 = Q * VV - (dt * rV2) * Pt[8];
                if (ro3 <= 0.0) {
                    ro3 = P.ro_floor;
                    nro++;
                }
                const double rro3 = 1.0 / ro3;
                const double u3 = (ro * u * VV - dt * (Pt[1] * rV2 - q1)) * rro3;
                const double v3 = (ro * v * VV - dt * ((Pt[2] - Sy * Am) * rV2 - q2)) * rro3;
                const double w3 = (ro * w * VV - dt * ((Pt[3] - Sphi * Am) * rV2)) * rro3;
                const double E = p / gm1 + ro * (u * u + v * v + w * w) * 0.5 + bb * i8p;
                const double E3 = E * VV - dt * (Pt[4] * rV2 - q3);
                const double bx3 = bx * VV - dt * (Pt[5] * rV2);
                const double by3 = by * VV - dt * (Pt[6] * rV2);
                const double bz3 = bz * VV - dt * ((Pt[7] - Sbz * Am) * rV2);
                double p3 = (E3 - 0.5 * ro3 * (u3 * u3 + v3 * v3 + w3 * w3) -
                             (bx3 * bx3 + by3 * by3 + bz3 * bz3) * i8p) *
                            gm1;
                if (p3 <= 0) {
                    p3 = P.p_floor;
                    npc++;
                }
                // pickup protons
                const double rp = e.f[kXro], pp = e.f[kXp], up = e.f[kXu], vp = e.f[kXv];
                double rp3 = rp * VV - dt * (Pt[9] * rV2);
                if (rp3 <= 0.0) {
                    rp3 = P.ro_floor;
                    nro++;
                }
                const double rrp3 = 1.0 / rp3;
                const double up3 = (rp * up * VV - dt * (Pt[10] * rV2)) * rrp3;
                const double vp3 = (rp * vp * VV - dt * ((Pt[11] - pp * Am) * rV2)) * rrp3;
                const double Ep = pp / gm1 + rp * (up * up + vp * vp) * 0.5;
                double pp3 = ((Ep * VV - dt * (Pt[12] * rV2)) - 0.5 * rp3 * (up3 * up3 + vp3 * vp3)) * gm1;
                if (pp3 <= 0) {
                    pp3 = P.p_floor;
                    npc++;
                }
                b.nxt[0][c] = ro3;
                b.nxt[1][c] = p3;
                b.nxt[2][c] = u3;
                b.nxt[3][c] = v3;
                b.nxt[4][c] = Q3;
                hnxt[kXw * nc + c] = w3;
                hnxt[kXbx * nc + c] = bx3;
                hnxt[kXby * nc + c] = by3;
                hnxt[kXbz * nc + c] = bz3;
                hnxt[kXro * nc + c] = rp3;
                hnxt[kXp * nc + c] = pp3;
                hnxt[kXu * nc + c] = up3;
                hnxt[kXv * nc + c] = vp3;
            } else {
                b.nxt[0][c] = par1.ro;
                b.nxt[1][c] = par1.p;
                b.nxt[2][c] = par1.u;
                b.nxt[3][c] = par1.v;
                b.nxt[4][c] = par1.Q;
#pragma unroll
                for (int k = 0; k < kMhdExtra; k++) hnxt[k * nc + c] = e.f[k];
            }
        }
    }
}

__global__ void __launch_bounds__(128, 6) mhd_update_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                         const double* __restrict__ fl,
                                                         const double* __restrict__ src,
                                                         const double* __restrict__ hcur, double* __restrict__ hnxt) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    double tmark = __longlong_as_double(0x7ff0000000000000LL);
    int nro = 0, npc = 0;
    if (c < d.n_cells) mhd_update_body(d, P, b, fl, src, hcur, hnxt, c, tmark, nro, npc);
    block_reduce_commit(tmark, nro, npc, 0, b.dt_acc, b.counters, b.status);
}

// ------------------------------------------------------------------ batched MHD step
// Many independent instances of the MHD + pickup step advance together: one
// launch per phase (surface tracking, rails, face units, cell update,
// commit) covers every instance.  A block finds its instance and first item
// in a static table (a block never straddles two instances, so the CFL
// block minimum goes to one instance's dt word) and copies the instance's
// descriptor into shared memory; the per-item work is the bodies of the
// one-instance kernels.
#ifndef GELIOS_BATCH_SMEM_DESC
#define GELIOS_BATCH_SMEM_DESC 0
#endif
#ifndef GELIOS_BATCH_FACE_MINB
#define GELIOS_BATCH_FACE_MINB 4
#endif
#ifndef GELIOS_BATCH_PLAIN_MINB
#define GELIOS_BATCH_PLAIN_MINB 4
#endif
#if GELIOS_BATCH_SMEM_DESC
#define BATCH_INSTANCE(I, e)          \
    __shared__ BatchInstance I;       \
    load_instance(I, t.inst + (e).x);
#else
#define BATCH_INSTANCE(I, e) const BatchInstance& I = t.inst[(e).x];
#endif
__device__ __forceinline__ void load_instance(BatchInstance& dst, const BatchInstance* __restrict__ src) {
    static_assert(sizeof(BatchInstance) % 16 == 0, "instance descriptor is copied as int4");
    const int4* s4 = reinterpret_cast<const int4*>(src);
    int4* d4 = reinterpret_cast<int4*>(&dst);
    for (int i = threadIdx.x; i < static_cast<int>(sizeof(BatchInstance) / 16); i += blockDim.x) d4[i] = s4[i];
    __syncthreads();
}

__global__ void __launch_bounds__(64) batch_surface_kernel(BatchTables t, int parity) {
    const int2 e = t.surf[blockIdx.x];
    BATCH_INSTANCE(I, e)
    const int j = e.y + (threadIdx.x >> 5);
    if (j >= I.d.n_lc + I.d.n_li + I.d.n_lo) return;
    surface_face_body(I.d, I.P, I.b[parity], I.surface, j, threadIdx.x & 31);
}

__global__ void __launch_bounds__(128) batch_rails_kernel(BatchTables t, int parity) {
    const int2 e = t.rails[blockIdx.x];
    BATCH_INSTANCE(I, e)
    rails_body(I.d, I.P, I.b[parity].dt_cur, I.surface, true, e.y);
}

// PLAIN: the plain interior group's tiles in the lean instance of the body,
// otherwise the other units'.  One generic launch for both took 628 us per
// step of 8 instances (1.32M cells, FP32 fluxes, ncu), these 334 and 100.
// Register caps of 160 or 96 instead of 128: 6% and 2% slower per step.
template <typename TF, bool PLAIN>
__global__ void __launch_bounds__(128, PLAIN ? GELIOS_BATCH_PLAIN_MINB : GELIOS_BATCH_FACE_MINB)
    batch_mhd_face_kernel(BatchTables t, int parity) {
    const int2 e = PLAIN ? t.plain[blockIdx.x] : t.units[blockIdx.x];
    BATCH_INSTANCE(I, e)
    const int u = e.y + threadIdx.x;
    const StepBuffers& b = I.b[parity];
    double tmin = __longlong_as_double(0x7ff0000000000000LL);
    int status = 0;
    if (u < (PLAIN ? I.d.u_c1 : I.d.n_units))
        tmin = mhd_face_body<TF, PLAIN>(I.d, I.P, I.M, b, I.hs[parity], I.fl, u, status);
    block_reduce_commit(tmin, 0, 0, status, b.dt_acc, b.counters, b.status);
}

__global__ void __launch_bounds__(128, 6) batch_mhd_update_kernel(BatchTables t, int parity) {
    const int2 e = t.cells[blockIdx.x];
    BATCH_INSTANCE(I, e)
    const int c = e.y + threadIdx.x;
    const StepBuffers& b = I.b[parity];
    double tmark = __longlong_as_double(0x7ff0000000000000LL);
    int nro = 0, npc = 0;
    if (c < I.d.n_cells) mhd_update_body(I.d, I.P, b, I.fl, I.src, I.hs[parity], I.hn[parity], c, tmark, nro, npc);
    block_reduce_commit(tmark, nro, npc, 0, b.dt_acc, b.counters, b.status);
}

__global__ void __launch_bounds__(256) batch_commit_kernel(BatchTables t, int parity) {
    const int2 e = t.points[blockIdx.x];
    BATCH_INSTANCE(I, e)
    const StepBuffers& b = I.b[parity];
    if (e.y == 0 && threadIdx.x == 0) {
        const unsigned long long a = *b.dt_acc;
        *b.dt_next = (a == 0x7ff0000000000000ULL) ? 100000000.0 : __longlong_as_double(static_cast<long long>(a));
        *b.dt_acc = 0x7ff0000000000000ULL;
    }
    const int i = e.y + threadIdx.x;
    if (i < I.d.n_points) {
        I.d.X[i] = I.d.X2[i];
        I.d.Y[i] = I.d.Y2[i];
    }
}

// `nsteps` batched MHD + pickup steps of every instance in ONE cooperative
// launch: the five phases of launch_batch_mhd_step (tracked-face speeds,
// rails, face units, cell update, commit) with a grid barrier where a kernel
// boundary was.  The blocks deal each phase's table by grid stride (table
// entries are equal-sized tiles of one instance each, so every CFL block
// minimum still goes to one instance's dt word); the per-item work is the
// bodies of the per-phase kernels, so a call leaves the same state as the
// same number of per-phase steps.  The grid must be co-resident (launched
// by cudaLaunchCooperativeKernel, which refuses a grid that is not).
template <typename TF>
__global__ void __launch_bounds__(128, GELIOS_BATCH_FACE_MINB) batch_mhd_persistent_kernel(BatchTables t, int nsteps) {
    cg::grid_group grid = cg::this_grid();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int st = 0; st < nsteps; st++) {
        const int parity = st & 1;
        // tracked faces: a surf entry holds two faces (one warp each), so a
        // 128-thread block takes two entries per round
        for (int i = 2 * blockIdx.x + (warp >> 1); i < t.n_surf; i += 2 * gridDim.x) {
            const int2 e = t.surf[i];
            const BatchInstance& I = t.inst[e.x];
            const int j = e.y + (warp & 1);
            if (j < I.d.n_lc + I.d.n_li + I.d.n_lo) surface_face_body(I.d, I.P, I.b[parity], I.surface, j, lane);
        }
        grid.sync();
        for (int i = blockIdx.x; i < t.n_rails; i += gridDim.x) {
            const int2 e = t.rails[i];
            const BatchInstance& I = t.inst[e.x];
            rails_body(I.d, I.P, I.b[parity].dt_cur, I.surface, true, e.y);
            __syncthreads();  // the next rail reuses the block's shared words
        }
        grid.sync();
        for (int i = blockIdx.x; i < t.n_plain + t.n_units; i += gridDim.x) {
            const bool plain = i < t.n_plain;
            const int2 e = plain ? t.plain[i] : t.units[i - t.n_plain];
            const BatchInstance& I = t.inst[e.x];
            const int u = e.y + threadIdx.x;
            const StepBuffers& b = I.b[parity];
            double tmin = __longlong_as_double(0x7ff0000000000000LL);
            int status = 0;
            if (u < (plain ? I.d.u_c1 : I.d.n_units)) tmin = mhd_face_body<TF>(I.d, I.P, I.M, b, I.hs[parity], I.fl, u, status);
            block_reduce_commit(tmin, 0, 0, status, b.dt_acc, b.counters, b.status);
            __syncthreads();  // the next tile reuses the reduction's shared words
        }
        grid.sync();
        for (int i = blockIdx.x; i < t.n_cells; i += gridDim.x) {
            const int2 e = t.cells[i];
            const BatchInstance& I = t.inst[e.x];
            const int c = e.y + threadIdx.x;
            const StepBuffers& b = I.b[parity];
            double tmark = __longlong_as_double(0x7ff0000000000000LL);
            int nro = 0, npc = 0;
            if (c < I.d.n_cells)
                mhd_update_body(I.d, I.P, b, I.fl, I.src, I.hs[parity], I.hn[parity], c, tmark, nro, npc);
            block_reduce_commit(tmark, nro, npc, 0, b.dt_acc, b.counters, b.status);
            __syncthreads();
        }
        grid.sync();
        // commit: a points entry covers 256 points (two per thread here)
        for (int i = blockIdx.x; i < t.n_points; i += gridDim.x) {
            const int2 e = t.points[i];
            const BatchInstance& I = t.inst[e.x];
            const StepBuffers& b = I.b[parity];
            if (e.y == 0 && threadIdx.x == 0) {
                const unsigned long long a = *b.dt_acc;
                *b.dt_next =
                    (a == 0x7ff0000000000000ULL) ? 100000000.0 : __longlong_as_double(static_cast<long long>(a));
                *b.dt_acc = 0x7ff0000000000000ULL;
            }
            for (int k = threadIdx.x; k < 256; k += blockDim.x) {
                const int p = e.y + k;
                if (p < I.d.n_points) {
                    I.d.X[p] = I.d.X2[p];
                    I.d.Y[p] = I.d.Y2[p];
                }
            }
        }
        grid.sync();
    }
}

// The dt / status words a call starts from: T[0] = T[1] = dt0, an empty CFL
// accumulator, zero clamp counters and status (layout: T[2], acc,
// counters[2], status, two more accumulators at byte 48).  A kernel rather than a copy from host memory: a
// copy from pageable memory would wait for the stream to drain.
__global__ void words_init_kernel(unsigned char* w, double dt0) {
    double* T = reinterpret_cast<double*>(w);
    unsigned long long* u = reinterpret_cast<unsigned long long*>(w + 16);
    T[0] = dt0;
    T[1] = dt0;
    u[0] = 0x7ff0000000000000ULL;
    u[1] = 0;
    u[2] = 0;
    *reinterpret_cast<int*>(w + 40) = 0;
    u[4] = 0x7ff0000000000000ULL;  // the plain form's second and third accumulators
    u[5] = 0x7ff0000000000000ULL;
}
__global__ void batch_words_init_kernel(BatchTables t, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const BatchInstance& I = t.inst[i];
    double* T = const_cast<double*>(I.b[0].dt_cur);  // T[0]; b[1].dt_cur is T[1]
    T[0] = I.P.dt0;
    T[1] = I.P.dt0;
    *I.b[0].dt_acc = 0x7ff0000000000000ULL;
    I.b[0].counters[0] = 0;
    I.b[0].counters[1] = 0;
    *I.b[0].status = 0;
}

// ------------------------------------------------------------------ residual
// L1 change of one state row between the two buffers: per block the sums
// of |a - b| and |a| in a fixed order, then one block adds the partials in
// block order (deterministic, no atomics).
__device__ __forceinline__ void residual_partial_body(const double* __restrict__ a, const double* __restrict__ b,
                                                      int n, double* __restrict__ part) {
    __shared__ double sd[256], sa[256];
    double dsum = 0.0, asum = 0.0;
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        dsum += fabs(a[i] - b[i]);
        asum += fabs(a[i]);
    }
    sd[threadIdx.x] = dsum;
    sa[threadIdx.x] = asum;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            sd[threadIdx.x] += sd[threadIdx.x + o];
            sa[threadIdx.x] += sa[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = sd[0];
        part[2 * blockIdx.x + 1] = sa[0];
    }
}
__device__ __forceinline__ void residual_final_body(const double* __restrict__ part, int nb, double* __restrict__ out) {
    double d = 0.0, s = 0.0;
    for (int k = 0; k < nb; k++) {
        d += part[2 * k];
        s += part[2 * k + 1];
    }
    out[0] = d;
    out[1] = s;
}
__global__ void __launch_bounds__(256) residual_partial_kernel(const double* __restrict__ a,
                                                               const double* __restrict__ b, int n,
                                                               double* __restrict__ part) {
    residual_partial_body(a, b, n, part);
}
__global__ void residual_final_kernel(const double* __restrict__ part, int nb, double* __restrict__ out) {
    residual_final_body(part, nb, out);
}
// The density residual of the active instances of a plain batch after an
// even number of steps, blockIdx.y the instance: the sums of
// residual_partial_kernel / residual_final_kernel per instance, gathered
// with its dt and status flags into four doubles for one read-back.
__global__ void __launch_bounds__(256) residual_batch_partial_kernel(const PlainInstance* __restrict__ inst,
                                                                     const int* __restrict__ active, int n,
                                                                     double* __restrict__ part) {
    const PlainInstance& I = inst[active[blockIdx.y]];
    residual_partial_body(I.b[0].cur[0], I.b[1].cur[0], n, part + static_cast<size_t>(kResidualScratch) * blockIdx.y);
}
__global__ void residual_batch_final_kernel(const PlainInstance* __restrict__ inst, const int* __restrict__ active,
                                            int nb, const double* __restrict__ part, double* __restrict__ out) {
    const PlainInstance& I = inst[active[blockIdx.x]];
    double* o = out + 4 * static_cast<size_t>(blockIdx.x);
    residual_final_body(part + static_cast<size_t>(kResidualScratch) * blockIdx.x, nb, o);
    o[2] = *I.b[0].dt_cur;
    o[3] = static_cast<double>(*I.b[0].status);
}

// ------------------------------------------------------------------ launchers
namespace {
inline int blocks_for(int n, int t) { return (n + t - 1) / t; }
}

void launch_centroid(const DevMesh& d, const double* X, const double* Y, double* cx, double* cy, double* rp,
                     double gamma, cudaStream_t s, double* vs, double* vol) {
    if (d.n_cells > 0)
        centroid_kernel<<<blocks_for(d.n_cells, 256), 256, 0, s>>>(d, X, Y, cx, cy, rp, 2 * gamma, vs, vol);
}
void launch_stationary_units(const DevMesh& d, const gelios_params& P, const StepBuffers& b, double* fl,
                             cudaStream_t s) {
    if (P.precision == GELIOS_PREC_FP32_FLUX)
        stationary32_unit_kernel<float><<<blocks_for(d.n_units, 128), 128, 0, s>>>(d, P, b, fl);
    else if (P.precision == GELIOS_PREC_FP32_WAVES)
        stationary_unit_kernel<WaveF32><<<blocks_for(d.n_units, 128), 128, 0, s>>>(d, P, b, fl);
    else
        stationary_unit_kernel<double><<<blocks_for(d.n_units, 128), 128, 0, s>>>(d, P, b, fl);
}
void launch_stationary_update(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const double* fl,
                              cudaStream_t s) {
    if (P.precision == GELIOS_PREC_FP32_FLUX)
        stationary32_update_kernel<<<blocks_for(d.n_cells, 128), 128, 0, s>>>(d, P, b, fl);
    else
        stationary_update_kernel<<<blocks_for(d.n_cells, 128), 128, 0, s>>>(d, P, b, fl);
}
// Lanes per block of the four-lanes-per-cell kernel, 0 where it does not take
// the grid: more faces than lanes, or more lanes than are resident at once.
// Where both take the grid the lanes are 3.6-4.5 times faster (see the
// kernel); 360 x 240 cells, beyond them: 35.2 us per step with three
// barriers, 21.9 in two phases with two.
static int plain_lane_threads(const DevMesh& d, int sms) {
    if (d.max_faces > 4 || !d.s_unit) return 0;
    const int64_t per = (4 * static_cast<int64_t>(d.n_cells) + sms - 1) / sms;
    const int64_t t = (per + 31) / 32 * 32;
    if (t > kLaneThreads) return 0;
    return t < 64 ? 64 : static_cast<int>(t);
}
cudaError_t launch_stationary_persistent(const DevMesh& d, const gelios_params& P, const StepBuffers& b0,
                                         const StepBuffers& b1, double* fl, int nsteps, cudaStream_t s) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    DevMesh dd = d;
    gelios_params pp = P;
    StepBuffers c0 = b0, c1 = b1;
    double* flp = fl;
    int n = nsteps;
    if (const int t = P.precision == GELIOS_PREC_FP32_FLUX ? 0 : plain_lane_threads(d, sms)) {
        const void* fn = P.precision == GELIOS_PREC_FP32_WAVES
                             ? reinterpret_cast<const void*>(&stationary_lanes_kernel<WaveF32>)
                             : reinterpret_cast<const void*>(&stationary_lanes_kernel<double>);
        void* args[] = {&dd, &pp, &c0, &c1, &n};
        const int64_t lanes = 4 * static_cast<int64_t>(d.n_cells);
        return cudaLaunchCooperativeKernel(fn, dim3(static_cast<unsigned>((lanes + t - 1) / t)), dim3(t), args, 0, s);
    }
    const void* fn = P.precision == GELIOS_PREC_FP32_FLUX
                         ? reinterpret_cast<const void*>(&stationary32_persistent_kernel<float>)
                     : P.precision == GELIOS_PREC_FP32_WAVES
                         ? reinterpret_cast<const void*>(&stationary_persistent_kernel<WaveF32>)
                         : reinterpret_cast<const void*>(&stationary_persistent_kernel<double>);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 128, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorCooperativeLaunchTooLarge;
    const int want = blocks_for(d.n_units > d.n_cells ? d.n_units : d.n_cells, 128);
    const int grid = want < per_sm * sms ? want : per_sm * sms;
    void* args[] = {&dd, &pp, &c0, &c1, &flp, &n};
    return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(128), args, 0, s);
}
__global__ void face_geometry_kernel(DevMesh d, double g2, const double* __restrict__ cx,
                                     const double* __restrict__ cy, double* __restrict__ upf) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= d.n_units) return;
    const int g = d.u_slot[u], K = d.u_cell[u];
    const int nb = d.u_twin[u] >= 0 ? d.snb[g] : -1;
    const int A = d.sA[g], B = d.sB[g];
    const FaceGeo f = face_geo(d.X[A], d.Y[A], d.X[B], d.Y[B], cx[K], cy[K], nb >= 0, nb >= 0 ? cx[nb] : 0.0,
                               nb >= 0 ? cy[nb] : 0.0);
    const size_t nu = d.n_units;
    upf[u] = pow2g(sqrt(f.f2), g2);
    double* geo = upf + nu;
    geo[u] = f.x2;
    geo[nu + u] = f.y2;
    geo[2 * nu + u] = f.n1;
    geo[3 * nu + u] = f.n2;
    geo[4 * nu + u] = f.f2;
    geo[5 * nu + u] = f.S;
    geo[6 * nu + u] = f.dist;
    geo[7 * nu + u] = f.distn;
}
__global__ void unit_geometry_kernel(DevMesh d, double gamma, double rad_stat, const double* __restrict__ cx,
                                     const double* __restrict__ cy, const double* __restrict__ rp,
                                     double* __restrict__ ugeo) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= d.n_units) return;
    const int g = d.u_slot[u], A = d.sA[g], B = d.sB[g];
    const UnitGeo f = unit_geo(gamma, rad_stat, d.u_info[u] & SI_TYPE_MASK, d.X[A], d.Y[A], d.X[B], d.Y[B], d.u_cell[u],
                               d.u_nb[u], cx, cy, rp);
    const size_t nu = d.n_units;
    const double rows[kUnitGeoRows] = {f.n1, f.n2, f.S,    f.dist, f.distn, f.kroO, f.kpO,
                                       f.CO, f.SO, f.kroN, f.kpN,  f.CN,    f.SN};
    for (int k = 0; k < kUnitGeoRows; k++) ugeo[k * nu + u] = rows[k];
    reinterpret_cast<uint32_t*>(ugeo + kUnitGeoRows * nu)[u] = f.flags;
}
void launch_unit_geometry(const DevMesh& d, const gelios_params& P, const double* cx, const double* cy,
                          const double* rp, double* ugeo, cudaStream_t s) {
    if (d.n_units <= 0) return;
    if (P.precision == GELIOS_PREC_FP32_FLUX)
        face_geometry_kernel<<<blocks_for(d.n_units, 128), 128, 0, s>>>(d, 2 * P.gamma, cx, cy, ugeo);
    else
        unit_geometry_kernel<<<blocks_for(d.n_units, 128), 128, 0, s>>>(d, P.gamma, P.rad_stat, cx, cy, rp, ugeo);
}
// FP32 fluxes: one cooperative grid for all instances.
static cudaError_t launch_stationary32_batch(const DevMesh& d, const PlainInstance* inst, const int* active,
                                             int n_active, int nsteps, cudaStream_t s) {
    const void* fn = reinterpret_cast<const void*>(&stationary32_batch_kernel<float>);
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 128, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorCooperativeLaunchTooLarge;
    const int64_t tiles = static_cast<int64_t>(n_active) * blocks_for(d.n_units > d.n_cells ? d.n_units : d.n_cells, 128);
    const int grid = tiles < static_cast<int64_t>(per_sm) * sms ? static_cast<int>(tiles) : per_sm * sms;
    DevMesh dd = d;
    const PlainInstance* ip = inst;
    const int* ap = active;
    int na = n_active, n = nsteps;
    void* args[] = {&dd, &ip, &ap, &na, &n};
    return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(128), args, 0, s);
}
// The launch of one cluster of `size` blocks per instance.  16 blocks need the
// non-portable size.
struct PlainClusters {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    const void* fn;
    PlainClusters(int n, int prec, int size) {
        fn = prec == GELIOS_PREC_FP32_WAVES ? reinterpret_cast<const void*>(&stationary_cluster_kernel<WaveF32>)
                                            : reinterpret_cast<const void*>(&stationary_cluster_kernel<double>);
        cfg.gridDim = dim3(static_cast<unsigned>(n) * size);
        cfg.blockDim = dim3(kClusterThreads);
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = size;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
    }
    PlainClusters(const PlainClusters&) = delete;
};
// More instances than are resident at size 1 run in waves (they are
// independent).
int plain_cluster_size(int n, int prec) {
    if (n <= 0 || prec == GELIOS_PREC_FP32_FLUX) return 0;
    for (int size = 16;; size /= 2) {
        PlainClusters c(n, prec, size);
        int fit = 0;
        if (cudaFuncSetAttribute(c.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&fit, c.fn, &c.cfg) != cudaSuccess) {  // a size the device does not offer
            cudaGetLastError();
            fit = 0;
        }
        if (fit >= n || size == 1) return size;
    }
}
cudaError_t launch_stationary_batch(const DevMesh& d, const PlainInstance* inst, const int* active, int n_active,
                                    int nsteps, int prec, int cluster_size, cudaStream_t s) {
    if (n_active <= 0 || nsteps <= 0) return cudaSuccess;
    if (prec == GELIOS_PREC_FP32_FLUX) return launch_stationary32_batch(d, inst, active, n_active, nsteps, s);
    PlainClusters c(n_active, prec, cluster_size);
    DevMesh dd = d;
    const PlainInstance* ip = inst;
    const int* ap = active;
    int n = nsteps;
    void* args[] = {&dd, &ip, &ap, &n};
    c.cfg.stream = s;
    return cudaLaunchKernelExC(&c.cfg, c.fn, args);
}
bool plain_batch_serial(const DevMesh& d, int n, int cluster_size) {
    int dev = 0, sms = 0;
    if (cluster_size <= 0 || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return plain_serial_faster(d.n_cells, n, plain_lane_threads(d, sms) > 0, cluster_size);
}
__global__ void plain_batch_words_init_kernel(const PlainInstance* inst, const int* active, int n) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const PlainInstance& I = inst[active[k]];
    double* T = const_cast<double*>(I.b[0].dt_cur);  // T[0]; b[1].dt_cur is T[1]
    T[0] = I.P.dt0;
    T[1] = I.P.dt0;
    for (int a = 0; a < 3; a++) *plain_acc(I.b[0].dt_acc, a) = 0x7ff0000000000000ULL;
    I.b[0].counters[0] = 0;
    I.b[0].counters[1] = 0;
    *I.b[0].status = 0;
}
void launch_plain_batch_words_init(const PlainInstance* inst, const int* active, int n, cudaStream_t s) {
    if (n > 0) plain_batch_words_init_kernel<<<blocks_for(n, 128), 128, 0, s>>>(inst, active, n);
}
void launch_mk2_recon(const DevMesh& d, const gelios_params& P, const StepBuffers& b, double* rec, cudaStream_t s) {
    const int nt = d.u_tr1 - d.u_tr0;
    if (nt > 0) mk2_recon_tracked_kernel<<<blocks_for(nt, 128), 128, 0, s>>>(d, P, b, rec);
}
// variant v of the tile kernel: threads per block x minimum resident blocks
// per SM (a register cap)
template <typename TF, int NT, int MINB>
static cudaError_t launch_tiles_v(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const TileView& t,
                                  const double* fl, const double* aux, cudaStream_t s) {
    const size_t smem = 5ull * static_cast<size_t>(t.max_slots) * sizeof(double);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(mk2_tile_kernel<TF, NT, MINB>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
    }
    mk2_tile_kernel<TF, NT, MINB><<<t.n_tiles, NT, smem, s>>>(d, P, b, t, fl, aux);
    return cudaGetLastError();
}
// Part 1 of a variant: the face units (none for the tile variants); part 2:
// the cell update (the whole tile kernel for the tile variants).  Part 1
// needs only the moved points; part 2 also the tracked-face fluxes and the
// source terms of the side stream.
template <typename TF, int MINB>
static void launch_faces_v(const DevMesh& d, const gelios_params& P, const StepBuffers& b, double* fl,
                           cudaStream_t s) {
    // the plain interior group in the variant's shape
    const int n0 = d.u_c1;
    if (n0 > 0) mk2_face_kernel<TF, MINB, false><<<blocks_for(n0, 128), 128, 0, s>>>(d, P, b, fl, n0);
}
// the plain interior group with the unit's gathers prefetched into L1
template <typename TF, int MINB>
static void launch_faces_pf(const DevMesh& d, const gelios_params& P, const StepBuffers& b, double* fl,
                            cudaStream_t s) {
    const int n0 = d.u_c1;
    if (n0 > 0) mk2_face_kernel<TF, MINB, true><<<blocks_for(n0, 128), 128, 0, s>>>(d, P, b, fl, n0);
}
// the C_1 interior and one-sided groups, each in an instance compiled for it
template <typename TF, bool PF>
static void launch_faces_rest(const DevMesh& d, const gelios_params& P, const StepBuffers& b, double* fl,
                              cudaStream_t s) {
    const int n1 = blocks_for(d.n_units - d.u_tr1, 128), nc = blocks_for(d.u_tr0 - d.u_c1, 128);
    if (n1 + nc > 0) mk2_face_rest_kernel<TF, 6, PF><<<n1 + nc, 128, 0, s>>>(d, P, b, fl, n1);
}
template <typename TF>
static cudaError_t launch_cells_p(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const TileView& t,
                                  double* fl, const double* aux, cudaStream_t s, int variant, int part) {
    if (variant >= 4 && variant < 8) {
        if (part != 2) return cudaSuccess;
        switch (variant) {
            case 4: return launch_tiles_v<TF, 256, 3>(d, P, b, t, fl, aux, s);
            case 5: return launch_tiles_v<TF, 256, 2>(d, P, b, t, fl, aux, s);
            case 6: return launch_tiles_v<TF, 128, 5>(d, P, b, t, fl, aux, s);
            default: return launch_tiles_v<TF, 128, 4>(d, P, b, t, fl, aux, s);
        }
    }
    if (part == 2) {
        mk2_update_kernel<kUpdAll><<<blocks_for(d.n_cells, 128), 128, 0, s>>>(d, P, b, fl, aux, nullptr, 0);
        return cudaGetLastError();
    }
    if (part == 3) {
        if (variant >= 8)
            launch_faces_rest<TF, true>(d, P, b, fl, s);
        else
            launch_faces_rest<TF, false>(d, P, b, fl, s);
        return cudaGetLastError();
    }
    switch (variant) {
        case 1: launch_faces_v<TF, 5>(d, P, b, fl, s); break;
        case 2: launch_faces_v<TF, 6>(d, P, b, fl, s); break;
        case 3: launch_faces_v<TF, 4>(d, P, b, fl, s); break;
        case 8: launch_faces_pf<TF, 8>(d, P, b, fl, s); break;
        case 9: launch_faces_pf<TF, 6>(d, P, b, fl, s); break;
        case 10: launch_faces_pf<TF, 4>(d, P, b, fl, s); break;
        default: launch_faces_v<TF, 8>(d, P, b, fl, s); break;
    }
    return cudaGetLastError();
}
const char* mk2_variant_name(int v) {
    static const char* names[kMk2Variants] = {"faces 128x8 + update",         "faces 128x5 + update",
                                              "faces 128x6 + update",         "faces 128x4 + update",
                                              "tiles 256x3",                  "tiles 256x2",
                                              "tiles 128x5",                  "tiles 128x4",
                                              "faces prefetched 128x8 + update", "faces prefetched 128x6 + update",
                                              "faces prefetched 128x4 + update"};
    return (v >= 0 && v < kMk2Variants) ? names[v] : "?";
}
int mk2_variant_launches(const DevMesh& d, int v, int part) {
    const bool tiles = v >= 4 && v < 8;
    if (part == 2) return 1;
    if (tiles) return 0;
    if (part == 1) return d.u_c1 > 0 ? 1 : 0;
    return d.u_tr0 > d.u_c1 || d.n_units > d.u_tr1 ? 1 : 0;
}
cudaError_t launch_mk2_cells(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const TileView& t,
                             double* fl, const double* aux, cudaStream_t s, int variant, int part) {
    if (P.precision == GELIOS_PREC_FP32_FLUX) return launch_cells_p<float>(d, P, b, t, fl, aux, s, variant, part);
    return launch_cells_p<double>(d, P, b, t, fl, aux, s, variant, part);
}
int launch_mk2_tracked_solve(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const double* rec,
                             double* pstar, cudaStream_t s) {
    const int nt = d.u_tr1 - d.u_tr0;
    if (nt <= 0) return 0;
    mk2_tracked_solve_kernel<<<blocks_for(nt, 2), 64, 0, s>>>(d, P, b, rec, pstar);
    return 1;
}
int launch_mk2_flux_tracked(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const double* rec,
                            const double* pstar, double* fl, cudaStream_t s) {
    const int nt = d.u_tr1 - d.u_tr0;
    if (nt <= 0) return 0;
    if (P.precision == GELIOS_PREC_FP32_FLUX)
        mk2_flux_tracked_kernel<float><<<blocks_for(nt, 32), 32, 0, s>>>(d, P, b, rec, fl, pstar);
    else
        mk2_flux_tracked_kernel<double><<<blocks_for(nt, 32), 32, 0, s>>>(d, P, b, rec, fl, pstar);
    return 1;
}
void launch_mk2_source(const DevMesh& d, const gelios_params& P, const StepBuffers& b, double* aux, cudaStream_t s) {
    if (d.n_cells > 0) mk2_source_kernel<<<blocks_for(d.n_cells, 128), 128, 0, s>>>(d, P, b, aux);
}
void launch_inner(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const int32_t* list, int n,
                  cudaStream_t s) {
    const int nb = blocks_for(n > 0 ? n : 1, 128);
    if (P.precision == GELIOS_PREC_FP32_FLUX)
        inner_cell_kernel<float><<<nb, 128, 0, s>>>(d, P, b, list, n);
    else
        inner_cell_kernel<double><<<nb, 128, 0, s>>>(d, P, b, list, n);
}
bool inner_lanes_ok(const DevMesh& d, const gelios_params& P, int n) {
    return P.precision != GELIOS_PREC_FP32_FLUX && d.max_faces <= 4 && n > 0 && n <= kInnerLaneCells;
}
cudaError_t launch_inner_lanes(const DevMesh& d, const gelios_params& P, const StepBuffers& b0, const StepBuffers& b1,
                               const int32_t* list, int n, double* tab, int nsteps, cudaStream_t s) {
    const void* fn = reinterpret_cast<const void*>(&inner_lanes_kernel<double>);
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 256, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorCooperativeLaunchTooLarge;
    const int lanes = 4 * n;
    int* itab = reinterpret_cast<int*>(tab + static_cast<size_t>(kInnerRows) * lanes);
    inner_table_kernel<<<blocks_for(lanes, 128), 128, 0, s>>>(d, P, b0, list, n, tab, itab);
    const int want = blocks_for(lanes, 256), most = per_sm * sms;
    const int rounds = blocks_for(want, most), grid = blocks_for(want, rounds);  // equal rounds
    DevMesh dd = d;
    gelios_params pp = P;
    StepBuffers c0 = b0, c1 = b1;
    int nn = n, ns = nsteps;
    void* args[] = {&dd, &pp, &c0, &c1, &list, &nn, &tab, &itab, &ns};
    return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(256), args, 0, s);
}
void launch_dt_finalize(const StepBuffers& b, cudaStream_t s) { dt_finalize_kernel<<<1, 1, 0, s>>>(b); }
void launch_commit(const DevMesh& d, const StepBuffers& b, cudaStream_t s, bool cap) {
    if (cap)
        commit_kernel<true><<<blocks_for(d.n_points > 0 ? d.n_points : 1, 256), 256, 0, s>>>(d, b);
    else
        commit_kernel<false><<<blocks_for(d.n_points > 0 ? d.n_points : 1, 256), 256, 0, s>>>(d, b);
}
void launch_mk2_update(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const double* fl,
                       const double* aux, cudaStream_t s, int mode, const int32_t* list, int n_list) {
    if (mode == kUpdEarly) {
        if (n_list > 0)
            mk2_update_kernel<kUpdEarly><<<blocks_for(n_list, 128), 128, 0, s>>>(d, P, b, fl, aux, list, n_list);
        return;
    }
    const int nb = blocks_for(d.n_cells, 128);
    if (mode == kUpdRest)
        mk2_update_kernel<kUpdRest><<<nb, 128, 0, s>>>(d, P, b, fl, aux, list, n_list);
    else if (mode == kUpdAllNoMark)
        mk2_update_kernel<kUpdAllNoMark><<<nb, 128, 0, s>>>(d, P, b, fl, aux, list, n_list);
    else
        mk2_update_kernel<kUpdAll><<<nb, 128, 0, s>>>(d, P, b, fl, aux, list, n_list);
}
void launch_rail_table(const DevMesh& d, int n_inner, cudaStream_t s) {
    const int nr = d.n_rail_a + d.n_rail_b + d.n_rail_c + d.n_rail_d;
    if (nr > 0)
        rail_table_kernel<<<nr, 128, 0, s>>>(d, n_inner, const_cast<double*>(d.rcs), const_cast<double*>(d.rsn),
                                             const_cast<double*>(d.rfrac));
}
int launch_motion(const DevMesh& d, const gelios_params& P, const StepBuffers& b, double* scratch, cudaStream_t s,
                  bool copy_outer_shock, const StepBuffers* fin) {
    int launches = 0;
    const int nf = d.n_lc + d.n_li + d.n_lo;
    if (nf > 0 || fin) {
        surface_faces_kernel<<<blocks_for(nf > 0 ? nf : 1, 2), 64, 0, s>>>(d, P, b, scratch, fin ? *fin : b,
                                                                            fin != nullptr);
        launches += 1;
    }
    const int nr = d.n_rail_a + d.n_rail_b + d.n_rail_c + d.n_rail_d;
    if (nr > 0) {
        rails_kernel<<<nr, 128, 0, s>>>(d, P, b.dt_cur, scratch, copy_outer_shock);
        launches++;
    }
    return launches;
}
void launch_hllc_batch(const gelios_params& P, int n, const double* in, double* out, cudaStream_t s) {
    hllc_batch_kernel<<<blocks_for(n, 128), 128, 0, s>>>(P, n, in, out);
}
int launch_k5_faces(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const double* hcur, double* fl,
                    cudaStream_t s, cudaStream_t s_c1, cudaStream_t s_rest) {
    const int nc1 = d.u_tr0 - d.u_c1, nt = d.u_tr1 - d.u_tr0, no = d.n_units - d.u_tr1;
    int n = 0;
    if (nt > 0) {  // first: the longest chain
        k5_tracked_kernel<<<blocks_for(nt, 2), 64, 0, s_rest>>>(d, P, b, hcur, fl);
        n++;
    }
    if (no > 0) {
        k5_face_kernel<kAnyGroup, 3><<<blocks_for(no, 128), 128, 0, s_rest>>>(d, P, b, hcur, fl, no);
        n++;
    }
    if (nc1 > 0) {
        k5_face_kernel<kC1Group, 4><<<blocks_for(nc1, 128), 128, 0, s_c1>>>(d, P, b, hcur, fl, nc1);
        n++;
    }
    if (d.u_c1 > 0) {
        k5_face_kernel<kPlainGroup, 5><<<blocks_for(d.u_c1, 128), 128, 0, s>>>(d, P, b, hcur, fl, d.u_c1);
        n++;
    }
    return n;
}
void launch_k5_update(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const double* fl,
                      const double* hcur, double* hnxt, cudaStream_t s) {
    k5_update_kernel<<<blocks_for(d.n_cells, 128), 128, 0, s>>>(d, P, b, fl, hcur, hnxt);
}
void launch_hlldq_batch(const gelios_params& P, int n, const double* in, double* out, cudaStream_t s) {
    hlldq_batch_kernel<<<blocks_for(n, 128), 128, 0, s>>>(P, n, in, out);
}
void launch_hlld_batch(const gelios_params& P, int n, const double* in, double* out, cudaStream_t s) {
    hlld_batch_kernel<<<blocks_for(n, 128), 128, 0, s>>>(P, n, in, out);
}
void launch_godunov_batch(const gelios_params& P, int n, const double* in, double* out, cudaStream_t s) {
    godunov_batch_kernel<<<blocks_for(n, 2), 64, 0, s>>>(P, n, in, out);
}
namespace {
// The plain interior group in the variant's shape on stream s, the other
// groups (a few percent of the units, every branch) in one fixed shape on
// stream sr (s itself, or a stream the caller forks and joins).
template <int BLOCK, int MINB>
void mhd_faces_shape(const DevMesh& d, const gelios_params& P, const gelios_mhd_params& M, const StepBuffers& b,
                     const double* hcur, double* fl, cudaStream_t s, cudaStream_t sr) {
    const int n0 = d.u_c1, nr = d.n_units - d.u_c1;
    const bool f32 = P.precision == GELIOS_PREC_FP32_FLUX;
    if (n0 > 0) {
        if (f32)
            mhd_face_kernel<float, BLOCK, MINB, true><<<blocks_for(n0, BLOCK), BLOCK, 0, s>>>(d, P, M, b, hcur, fl);
        else
            mhd_face_kernel<double, BLOCK, MINB, true><<<blocks_for(n0, BLOCK), BLOCK, 0, s>>>(d, P, M, b, hcur, fl);
    }
    if (nr > 0) {
        if (f32)
            mhd_face_kernel<float, 128, 3, false><<<blocks_for(nr, 128), 128, 0, sr>>>(d, P, M, b, hcur, fl);
        else
            mhd_face_kernel<double, 128, 3, false><<<blocks_for(nr, 128), 128, 0, sr>>>(d, P, M, b, hcur, fl);
    }
}
}  // namespace

const char* mhd_face_variant_name(int v) {
    static const char* names[kMhdFaceVariants] = {"128x3", "128x1", "128x4", "64x6", "64x3", "256x1"};
    return (v >= 0 && v < kMhdFaceVariants) ? names[v] : "?";
}
int launch_mhd_faces(const DevMesh& d, const gelios_params& P, const gelios_mhd_params& M, const StepBuffers& b,
                     const double* hcur, double* fl, cudaStream_t s, int variant, cudaStream_t s_rest) {
    if (d.n_units <= 0) return 0;
    cudaStream_t sr = s_rest ? s_rest : s;
    switch (variant) {
        case 1: mhd_faces_shape<128, 1>(d, P, M, b, hcur, fl, s, sr); break;
        case 2: mhd_faces_shape<128, 4>(d, P, M, b, hcur, fl, s, sr); break;
        case 3: mhd_faces_shape<64, 6>(d, P, M, b, hcur, fl, s, sr); break;
        case 4: mhd_faces_shape<64, 3>(d, P, M, b, hcur, fl, s, sr); break;
        case 5: mhd_faces_shape<256, 1>(d, P, M, b, hcur, fl, s, sr); break;
        default: mhd_faces_shape<128, 3>(d, P, M, b, hcur, fl, s, sr); break;
    }
    return (d.u_c1 > 0 ? 1 : 0) + (d.n_units > d.u_c1 ? 1 : 0);
}
// Frozen-grid residual of the moving-grid operator, per block: over the
// cells that take part in a step (centroid radius >= R11, not C_centr) the
// sum of |sum of the mass fluxes F.S of the cell's face slots| / rotated
// volume (the density change per unit time the step's flux balance gives
// with the grid held still: d(rho V)/dt = -sum F.S, Setka.cpp:10425-10431),
// and the sum of |rho| over every cell.  Fixed-order tree sums.
__global__ void __launch_bounds__(256) op_residual_partial_kernel(DevMesh d, gelios_params P, StepBuffers b,
                                                                  const double* __restrict__ fl,
                                                                  double* __restrict__ part) {
    __shared__ double sd[256], sa[256];
    double dsum = 0.0, asum = 0.0;
    for (int c = blockIdx.x * 256 + threadIdx.x; c < d.n_cells; c += gridDim.x * 256) {
        asum += fabs(b.cur[0][c]);
        const double x = b.cx[c], y = b.cy[c];
        if (sqrt(sq(x) + sq(y)) < P.R11 || (d.cflags[c] & CF_CENTR)) continue;
        double pt = 0.0;
        for (int g = d.gstart[c]; g < d.gstart[c + 1]; g++) pt = pt + unit_flux(fl, d.s_unit[g]);
        dsum += fabs(pt) / b.vol[c];
    }
    sd[threadIdx.x] = dsum;
    sa[threadIdx.x] = asum;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            sd[threadIdx.x] += sd[threadIdx.x + o];
            sa[threadIdx.x] += sa[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = sd[0];
        part[2 * blockIdx.x + 1] = sa[0];
    }
}
int launch_op_residual(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const double* fl,
                       double* scratch, cudaStream_t s) {
    const int n = d.n_cells;
    const int nb = n > 0 ? (blocks_for(n, 256) < 296 ? blocks_for(n, 256) : 296) : 1;
    op_residual_partial_kernel<<<nb, 256, 0, s>>>(d, P, b, fl, scratch + 2);
    residual_final_kernel<<<1, 1, 0, s>>>(scratch + 2, nb, scratch);
    return 2;
}
int launch_residual(const double* a, const double* b, int n, double* scratch, cudaStream_t s) {
    const int nb = n > 0 ? (blocks_for(n, 256) < 296 ? blocks_for(n, 256) : 296) : 1;
    residual_partial_kernel<<<nb, 256, 0, s>>>(a, b, n, scratch + 2);
    residual_final_kernel<<<1, 1, 0, s>>>(scratch + 2, nb, scratch);
    return 2;
}
void launch_residual_batch(const PlainInstance* inst, const int* active, int n_active, int n_cells, double* part,
                           double* out, cudaStream_t s) {
    int nb = blocks_for(n_cells, 256);
    if (nb > 296) nb = 296;
    if (nb < 1) nb = 1;
    for (int i = 0; i < n_active; i += 65535) {  // a grid's y extent
        const int k = n_active - i < 65535 ? n_active - i : 65535;
        residual_batch_partial_kernel<<<dim3(nb, k), 256, 0, s>>>(inst, active + i, n_cells,
                                                                  part + static_cast<size_t>(kResidualScratch) * i);
    }
    residual_batch_final_kernel<<<n_active, 1, 0, s>>>(inst, active, nb, part, out);
}
void launch_words_init(void* words, double dt0, cudaStream_t s) {
    words_init_kernel<<<1, 1, 0, s>>>(static_cast<unsigned char*>(words), dt0);
}
void launch_batch_words_init(const BatchTables& t, int n, cudaStream_t s) {
    if (n > 0) batch_words_init_kernel<<<blocks_for(n, 128), 128, 0, s>>>(t, n);
}
cudaError_t launch_batch_mhd_step(const BatchTables& t, int parity, cudaStream_t s, cudaStream_t s_rest,
                                  cudaEvent_t fork, cudaEvent_t join) {
    if (t.n_surf > 0) batch_surface_kernel<<<t.n_surf, 64, 0, s>>>(t, parity);
    if (t.n_rails > 0) batch_rails_kernel<<<t.n_rails, 128, 0, s>>>(t, parity);
    cudaError_t e = cudaEventRecord(fork, s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s_rest, fork, 0);
    if (e != cudaSuccess) return e;
    if (t.n_units > 0) {
        if (t.fp32)
            batch_mhd_face_kernel<float, false><<<t.n_units, 128, 0, s_rest>>>(t, parity);
        else
            batch_mhd_face_kernel<double, false><<<t.n_units, 128, 0, s_rest>>>(t, parity);
    }
    if (t.n_plain > 0) {
        if (t.fp32)
            batch_mhd_face_kernel<float, true><<<t.n_plain, 128, 0, s>>>(t, parity);
        else
            batch_mhd_face_kernel<double, true><<<t.n_plain, 128, 0, s>>>(t, parity);
    }
    e = cudaEventRecord(join, s_rest);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s, join, 0);
    if (e != cudaSuccess) return e;
    if (t.n_cells > 0) batch_mhd_update_kernel<<<t.n_cells, 128, 0, s>>>(t, parity);
    if (t.n_points > 0) batch_commit_kernel<<<t.n_points, 256, 0, s>>>(t, parity);
    return cudaSuccess;
}
cudaError_t launch_batch_mhd_persistent(const BatchTables& t, int nsteps, int blocks_per_sm, cudaStream_t s,
                                        int* max_per_sm) {
    const void* fn = t.fp32 ? reinterpret_cast<const void*>(&batch_mhd_persistent_kernel<float>)
                            : reinterpret_cast<const void*>(&batch_mhd_persistent_kernel<double>);
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 128, 0);
    if (e != cudaSuccess) return e;
    if (max_per_sm) *max_per_sm = per_sm;
    if (per_sm < 1 || blocks_per_sm > per_sm) return cudaErrorCooperativeLaunchTooLarge;
    if (nsteps <= 0) return cudaSuccess;
    const int k = blocks_per_sm > 0 ? blocks_per_sm : per_sm;
    BatchTables tt = t;
    int n = nsteps;
    void* args[] = {&tt, &n};
    return cudaLaunchCooperativeKernel(fn, dim3(k * sms), dim3(128), args, 0, s);
}
void launch_mhd_update(const DevMesh& d, const gelios_params& P, const StepBuffers& b, const double* fl,
                       const double* src, const double* hcur, double* hnxt, cudaStream_t s) {
    mhd_update_kernel<<<blocks_for(d.n_cells, 128), 128, 0, s>>>(d, P, b, fl, src, hcur, hnxt);
}

}  // namespace gelios
