// The trajectory tracer: kernels/trace_trajectories_2d/trace_trajectories_2d_pyccel.py:42-507
// re-designed for the B200.
//
// One thread per live trajectory advances it by at most `window` steps per launch (RK4 or
// Boris's kick-drift-kick through the staggered edge fields of the patches, plane
// crossings, kept paths, exit and electrode sub-cell tests: the reference's step, term by
// term, in FP64 with no contracted multiply-add, so a trajectory ends bit for bit where the
// reference's CPU kernel ends it; the only fused multiply-adds are those of `div_known` and
// `Num`, whose quotients and roots are the IEEE operations').  Instead of adding its charge
// to the mesh with atomics, every step writes one deposit record (cell, u, w, dq dt) to a
// slot fixed by (window, step, trajectory); between windows the live trajectories are
// compacted in order, and the records are sorted by cell and reduced per cell in record order
// (deposit.cu), so the node charges are deterministic.  The deposits run on a side stream under the next
// windows, in the order the record buffers were filled.  Short windows bound the tail of a
// warp (its threads wait only for the longest trajectory of the window, not of the whole
// trace).
#include <algorithm>

#include "common.cuh"

namespace bt {

namespace {

struct Trace {
    bt_trace_args a;
    i64 nx, ny;       // the last patch's node counts
    bt_magnetic mag;  // the magnetic field of the MAG kernels
    // A batch of candidate meshes (the BATCH kernels): every trajectory's candidate, and
    // where each candidate's cell table starts in a.cells.  Row c of a.patch_int /
    // a.patch_real is candidate c's one patch (shape, offsets, origin, spacing, extent).
    const int32_t *cand;
    const i64 *cell_off;
    // the candidates' electrode shapes (candidate c's: shape_first[c] .. shape_first[c + 1]
    // - 1 of `shapes`), or shape_first NULL: pause for the caller's test
    const i64 *shape_first;
    Shapes shapes;
};

// The cell of x on a graded axis: the last node at or before x, within the axis (0 left of
// it or for a NaN).  `hint` is where the search starts: a trajectory's points lie in its last
// cell or beside it, so the walk reads two or three nodes where a bisection reads eleven
// of 1025, each waiting for the one before.
__device__ __forceinline__ int node_cell(double x, const double *__restrict__ nodes, int n,
                                         int hint) {
    if (!(x > nodes[0])) return 0;
    if (x >= nodes[n - 1]) return n - 2;
    int c = hint;
    while (x < nodes[c]) --c;
    while (x >= nodes[c + 1]) ++c;
    return c;
}

// The same by bisection, for a window's first point, which has no cell to walk from.
__device__ __forceinline__ int first_cell(double x, const double *__restrict__ nodes, int n) {
    int lo = 0, hi = n - 1;
    while (hi - lo > 1) {
        const int mid = (lo + hi) / 2;
        if (nodes[mid] <= x)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

__device__ __forceinline__ i64 finest_patch(const bt_trace_args &a, i64 P, double px, double py) {
    for (i64 qq = 0; qq < P - 1; ++qq) {
        const double *pr = a.patch_real + qq * 7;
        if (px >= __ldg(pr + 3) && px <= __ldg(pr + 5) && py >= __ldg(pr + 4) &&
            py <= __ldg(pr + 6))
            return qq;
    }
    return P - 1;
}

// A patch's shape: node counts, its offsets into the edge-field and node arrays, origin and
// spacing (one row of patch_int / patch_real), and the spacing's reciprocal for `div_known`
// (0: divide plainly).
struct PatchGeom {
    i64 pnx, pny, ofx, ofy, ofn;
    double pox, poy, phh, rphh;
};

__device__ __forceinline__ PatchGeom patch_geom(const bt_trace_args &a, i64 pp) {
    const i64 *pi = a.patch_int + pp * 6;
    const double *pr = a.patch_real + pp * 7;
    return {__ldg(pi + 0), __ldg(pi + 1), __ldg(pi + 2), __ldg(pi + 3), __ldg(pi + 5),
            __ldg(pr + 0), __ldg(pr + 1), __ldg(pr + 2), 0.0};
}

// Cell indices are 32-bit: a patch has fewer than 2^31 nodes along an axis (the deposit keys
// are 32-bit).  floor and truncation saturate outside that range, where the clamps that
// follow them give what the 64-bit conversions give.
__device__ __forceinline__ int clamp_index(int i, int lo, int hi) { return min(max(i, lo), hi); }

// The cell i of s among cells 0 .. last and the weight w in it.
__device__ __forceinline__ int cell_weight(double s, int last, double &w) {
    const int i = clamp_index(__double2int_rd(s), 0, last);
    w = s - (double)i;
    return i;
}

__device__ __forceinline__ double bilinear(const double *__restrict__ f, int stride, double u,
                                           double w) {
    const double f00 = __ldg(f), f01 = __ldg(f + 1);
    const double f10 = __ldg(f + stride), f11 = __ldg(f + stride + 1);
    const double low = f00 + w * (f01 - f00);
    const double high = f10 + w * (f11 - f10);
    return low + u * (high - low);
}

// E at the point (sx, sy) in cells of patch g from its origin (the finest patch holding the
// point; trace_trajectories_2d_pyccel.py:212-269).  The straight-line form takes the cell of
// s + 1/2 from the cell c of s -- it is c, or c + 1 where s + 1/2, as rounded, has reached
// it -- without a second pair of conversions but for a point past the mesh's edge, whose cells
// are clamped.  (Every trajectory that leaves has such a point in its last step; called odd,
// it made the whole warp take a step with IEEE operations, one warp step in ten of 100,000
// short trajectories on a planar 81 x 31 mesh with boxes: 6.8 ms of windows for 4.9, or 5.2
// with IEEE operations throughout.)
template <class N>
__device__ __forceinline__ void edge_field_cells(N &num, const bt_trace_args &a,
                                                 const PatchGeom &g, double sx, double sy,
                                                 double &ex, double &ey) {
    const int pnx = (int)g.pnx, pny = (int)g.pny;
    const double hx = sx + 0.5, hy = sy + 0.5;
    int ix, jx, iy, jy;
    double ux, wx, uy, wy;
    if (N::fast) {
        const int i = __double2int_rd(sx), j = __double2int_rd(sy);
        const double fi = (double)i, fj = (double)j;
        const bool up_i = hx >= fi + 1.0, up_j = hy >= fj + 1.0;
        ix = clamp_index(clamp_index(i, -1, pnx - 1) + (up_i ? 1 : 0), 0, pnx - 1);
        jx = clamp_index(j, 0, pny - 2);
        iy = clamp_index(i, 0, pnx - 2);
        jy = clamp_index(clamp_index(j, -1, pny - 1) + (up_j ? 1 : 0), 0, pny - 1);
        uy = sx - fi;
        wx = sy - fj;
        ux = hx - (up_i ? fi + 1.0 : fi);
        wy = hy - (up_j ? fj + 1.0 : fj);
        if (iy != i || jx != j) {
            ux = hx - (double)ix;
            wx = sy - (double)jx;
            uy = sx - (double)iy;
            wy = hy - (double)jy;
        }
    } else {
        ix = cell_weight(hx, pnx - 1, ux);
        jx = cell_weight(sy, pny - 2, wx);
        iy = cell_weight(sx, pnx - 2, uy);
        jy = cell_weight(hy, pny - 1, wy);
    }
    ex = bilinear(a.fxs + g.ofx + (i64)ix * pny + jx, pny, ux, wx);
    ey = bilinear(a.fys + g.ofy + (i64)iy * (pny + 1) + jy, pny + 1, uy, wy);
}

// (B_z, B_r) of an on-axis profile at axial position z and radius r (fields.py:250-279,
// term by term: the derivatives interpolated between samples, then the series in r); rhz
// the reciprocal of the samples' spacing.
template <class N>
__device__ __forceinline__ void axial_field(N &num, const bt_magnetic &m, double rhz, double z,
                                            double r, double &bz_out, double &br_out) {
    const i64 n = m.n;
    const int K = m.order + 1;
    const double s = num.known(z - m.z0, m.hz, rhz);
    i64 i = (i64)__double2int_rd(s);
    if (i < 3)
        i = 3;
    else if (i > n - 5)
        i = n - 5;
    const double t = s - (double)i;
    const double *lo = m.samples + i * K, *hi = lo + K;
    double d[7];
#pragma unroll
    for (int k = 0; k < 7; ++k)
        if (k < K) {
            const double a = __ldg(lo + k);
            d[k] = a + t * (__ldg(hi + k) - a);
        }
    const double r2 = r * r;
    const double bz_c[4] = {1.0, -1.0 / 4.0, 1.0 / 64.0, -1.0 / 2304.0};
    const double br_c[3] = {-1.0 / 2.0, 1.0 / 16.0, -1.0 / 384.0};
    double bz = d[0], br = 0.0, power = 1.0;
#pragma unroll
    for (int k = 1; k <= 3; ++k)
        if (k <= m.order / 2) {
            power = power * r2;
            bz = bz + bz_c[k] * power * d[2 * k];
        }
    power = r;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        if (k < (m.order + 1) / 2) {
            br = br + br_c[k] * power * d[2 * k + 1];
            power = power * r2;
        }
    bz_out = bz;
    br_out = br;
}

// The Cartesian B at (q0, q1, q2): mode 1 on a cylindrical mesh ((cy, cz) the radial unit
// vector, r the radius), mode 2 a planar mesh with the solenoid axis on y = axis_y.
template <class N>
__device__ __forceinline__ void magnetic_at(N &num, const bt_magnetic &m, double rhz, double q0,
                                            double q1, double r, double cy, double cz, double *b) {
    double bz, br;
    if (m.mode == 1) {
        axial_field(num, m, rhz, q0, r, bz, br);
        b[0] = bz;
        b[1] = br * cy;
        b[2] = br * cz;
    } else {
        const double yr = q1 - m.axis_y;
        axial_field(num, m, rhz, q0, fabs(yr), bz, br);
        b[0] = bz;
        b[1] = yr < 0.0 ? -br : br;
        b[2] = 0.0;
    }
}

// v <- Boris's kick over tau in the fields e, b (non-relativistic; tracer.py:605-621):
// v- = v + (tau/2) q/m E, t = (tau/2) q/m B, v+ = v- + (v- + v- x t) x 2t / (1 + t^2),
// then + (tau/2) q/m E; the operations in the oracle's order.
template <class N>
__device__ __forceinline__ void kick(N &num, double *v, const double *e, const double *b,
                                     double tau, double qm) {
    const double f = 0.5 * tau * qm;
    const double m0 = v[0] + f * e[0], m1 = v[1] + f * e[1], m2 = v[2] + f * e[2];
    const double t0 = f * b[0], t1 = f * b[1], t2 = f * b[2];
    const double d = num.div_sound(2.0, 1.0 + (t0 * t0 + t1 * t1 + t2 * t2));
    const double s0 = d * t0, s1 = d * t1, s2 = d * t2;
    const double p0 = m0 + (m1 * t2 - m2 * t1);
    const double p1 = m1 + (m2 * t0 - m0 * t2);
    const double p2 = m2 + (m0 * t1 - m1 * t0);
    const double w0 = m0 + (p1 * s2 - p2 * s1);
    const double w1 = m1 + (p2 * s0 - p0 * s2);
    const double w2 = m2 + (p0 * s1 - p1 * s0);
    v[0] = w0 + f * e[0];
    v[1] = w1 + f * e[1];
    v[2] = w2 + f * e[2];
}

// 1 / gamma of a proper velocity: exactly 1 without relativity (inv_c2 = 0), which the
// non-general kernels fold away.
template <bool GENERAL, class N>
__device__ __forceinline__ double inv_gamma(N &num, double u0, double u1, double u2,
                                            double inv_c2) {
    return GENERAL ? num.div_sound(1.0, num.root(1.0 + (u0 * u0 + u1 * u1 + u2 * u2) * inv_c2))
                   : 1.0;
}

// What a trajectory's steps share: its mesh (its candidate's in a batch), its base patch,
// the spacings' reciprocals, its charge over mass and its current.
struct Geo {
    double ox, oy, h, rh, rhz;
    PatchGeom base;
    double qm, dq, fraction, inv_c2;
    int P, n_x_nodes;
    bool graded;
    bool same;  // one patch, which is the mesh: cell coordinates serve both
    bool fast;  // the straight-line arithmetic may be tried (every reciprocal is one, the
                // origins are sound)
};

// A point on the mesh: its radius or distance from the axis (the mesh's second coordinate)
// with the root's reciprocal, its uniform x, its cell on a graded axis, its cell coordinates.
struct Place {
    double r, y, lx, sx, sy;
    int cell;
};

// The state of a trajectory between steps: position, velocity, place, and the pace it sets --
// the local spacing, the speed's square and the spacing over the speed (-1 at rest) -- with
// Boris the fields at the last step's end (q/m E, or E and B).
struct State {
    double x[3], v[3];
    Place at;
    double gv, hloc, speed2, dt0;
    double e[3], b[3];
    bool have;
};

// A step's deposit: the shares of the four nodes of its midpoint's cell.
struct Share {
    uint32_t key;
    double c00, c01, c10, c11;
};

// x on the uniform axis (its own value on a mesh that is not graded), its graded cell found
// from `hint` on.
template <bool GENERAL, class N>
__device__ __forceinline__ double uniform_x(N &num, const bt_trace_args &a, const Geo &G, double x,
                                            int hint, int &cell) {
    cell = hint;
    if (!GENERAL || !G.graded) return x;
    const double *nodes = a.x_nodes;
    const int c = cell = node_cell(x, nodes, G.n_x_nodes, hint);
    return G.ox + G.h * ((double)c + num.div(x - nodes[c], nodes[c + 1] - nodes[c]));
}

template <int CYL, bool GENERAL, class N>
__device__ __forceinline__ void locate(N &num, const bt_trace_args &a, const Geo &G,
                                       const double *q, int hint, Place &W) {
    W.y = 0.0;
    W.r = q[1];
    if (CYL == 1)
        W.r = num.root(q[1] * q[1] + q[2] * q[2], W.y);
    else if (CYL == 2)
        W.r = G.oy + fabs(q[1] - G.oy);
    W.lx = uniform_x<GENERAL>(num, a, G, q[0], hint, W.cell);
    // (the coordinates tested, not their differences from the origin; a radius is its root's)
    num.not_tiny(W.lx);
    if (CYL != 1) num.not_tiny(W.r);
    W.sx = num.known_sound(W.lx - G.ox, G.h, G.rh);
    W.sy = num.known_sound(W.r - G.oy, G.h, G.rh);
}

// The pace of a state at its place.
template <bool GENERAL, bool MAG, class N>
__device__ __forceinline__ void set_pace(N &num, const bt_trace_args &a, const Geo &G, State &S) {
    double hloc = G.h;
    if (GENERAL) {
        for (int qq = 0; qq < G.P - 1; ++qq) {
            const double *pr = a.patch_real + qq * 7;
            if (S.at.lx >= __ldg(pr + 3) && S.at.lx <= __ldg(pr + 5) && S.at.r >= __ldg(pr + 4) &&
                S.at.r <= __ldg(pr + 6)) {
                hloc = __ldg(pr + 2);
                break;
            }
        }
        if (G.graded) {
            const double dxc = a.x_nodes[S.at.cell + 1] - a.x_nodes[S.at.cell];
            if (MAG) {
                // the NumPy tracer's spacing: the smaller of the cell's edge and h
                if (dxc < hloc) hloc = dxc;
            } else {
                const double d2 = num.known(dxc, G.h, G.rh);
                if (d2 < 1.0) hloc = hloc * d2;
            }
        }
    }
    S.hloc = hloc;
    const double s = S.v[0] * S.v[0] + S.v[1] * S.v[1] + S.v[2] * S.v[2];
    double y;
    const double root = num.root(s, y);
    const double speed = GENERAL ? S.gv * root : root;
    S.speed2 = speed * speed;
    // (at rest the quotient is not used; Num<true> then calls the step odd)
    const double time =
        GENERAL ? num.div(hloc, speed) : num.over_sound(hloc, speed, num.inverse(speed, y));
    S.dt0 = speed > 0.0 ? time : -1.0;
}

// E and, with MAG, B at the point q located at W.
template <int CYL, bool GENERAL, bool MAG, class N>
__device__ __forceinline__ void fields_at(N &num, const bt_trace_args &a, const bt_magnetic &mag,
                                          const Geo &G, const double *q, const Place &W, double *E,
                                          double *B) {
    double cy = 0.0, cz = 0.0;
    if (CYL == 1) {
        // (selected, not branched around: with Num<true> the quotients cost no branch)
        const bool off_axis = W.r > 0.0;
        const double ir = num.inverse(W.r, W.y);
        const double uy = num.over(q[1], W.r, ir), uz = num.over(q[2], W.r, ir);
        cy = off_axis ? uy : 0.0;
        cz = off_axis ? uz : 0.0;
    } else if (CYL == 2) {
        cy = 1.0;
        if (q[1] < G.oy) cy = -1.0;
    }
    double ex, ey;
    if ((N::fast && !GENERAL) || G.same) {  // (the straight-line form is for G.same only)
        edge_field_cells(num, a, G.base, W.sx, W.sy, ex, ey);
    } else {
        const PatchGeom g = GENERAL ? patch_geom(a, finest_patch(a, G.P, W.lx, W.r)) : G.base;
        edge_field_cells(num, a, g, num.div(W.lx - g.pox, g.phh), num.div(W.r - g.poy, g.phh), ex,
                         ey);
    }
    E[0] = ex;
    if (CYL != 0) {
        E[1] = ey * cy;
        E[2] = ey * cz;
    } else {
        E[1] = ey;
        E[2] = 0.0;
    }
    if (MAG) magnetic_at(num, mag, G.rhz, q[0], q[1], W.r, cy, cz, B);
}

// g = q/m (E + u x B) (tracer.py:519-529), or q/m E.
template <bool MAG>
__device__ __forceinline__ void pull(double qm, const double *E, const double *B, const double *u,
                                     double *g) {
    if (MAG) {
        g[0] = qm * (E[0] + (u[1] * B[2] - u[2] * B[1]));
        g[1] = qm * (E[1] + (u[2] * B[0] - u[0] * B[2]));
        g[2] = qm * (E[2] + (u[0] * B[1] - u[1] * B[0]));
    } else {
        g[0] = qm * E[0];
        g[1] = qm * E[1];
        g[2] = qm * E[2];
    }
}

// One step from S to T and its deposit in D; the rounding of every operation is the
// reference's.  The forms but kIeee: straight-line arithmetic (Num<true>), false where it may
// not hold -- the caller steps again with kIeee.
//
// kSpeculated also takes the step as limited by the speed, whose time the step before has left
// in S.dt0, and only checks that the acceleration would not shorten it (`limited` where it
// may), with a margin of 1e-9 against rounding: |a| < 2 v^2 / h, all squared, no root or
// quotient.  So the time does not wait for the first field: the points of the second stage
// (x + dt/2 v) and of the first are looked up together, as are those of the third (which
// needs the first stage's field) and the fourth (the second's), the chain of a Runge-Kutta
// step two lookups long instead of four with the step time's two roots and quotient between.  A step limited by the
// acceleration (a beam starting nearly at rest, or turning back) is taken again as kTimed,
// which waits for the field: 100,000 ions turned back at points of their own in a 41 x 21
// mesh take 1.69 ms (planar 1.44), as kIeee 2.07 (1.56); all steps so, 1.72 (1.34).  (A loop
// around the straight-line step in kTimed's place cost the other traces 7 %.)
//
// Bound by latency still: one warp a scheduler on 20,000 rings, 1,013 instructions of 500 in
// FP64 a step (8 cycles each behind another, 2 of issue).  A window of 64 Runge-Kutta steps of
// 20,000 rings at 801 x 201 takes 132 us (216 with IEEE roots and quotients and a step time
// that waits for the field); 64 Boris steps of 100,000 ions on a graded 1025 x 513 mesh in
// a solenoid 965 us before, 465 now (a pass's 68 windows on average).
enum StepForm { kIeee = 0, kSpeculated = 1, kTimed = 2 };

template <int CYL, int INTEG, bool GENERAL, bool MAG, StepForm FORM>
__device__ __forceinline__ bool advance(const bt_trace_args &a, const bt_magnetic &mag,
                                        const Geo &G, const State &S, State &T, Share &D,
                                        bool &limited) {
    Num<FORM != kIeee> num;
    const double qm = G.qm, inv_c2 = G.inv_c2;
    const double gv = GENERAL ? S.gv : 1.0;
    double E[3], B[3] = {0.0, 0.0, 0.0}, a1[3];
    if (INTEG != 0 && S.have) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            E[c] = S.e[c];
            if (MAG) B[c] = S.b[c];
        }
    } else {
        fields_at<CYL, GENERAL, MAG>(num, a, mag, G, S.x, S.at, E, B);
    }
    if (INTEG != 0 && !MAG && S.have) {
#pragma unroll
        for (int c = 0; c < 3; ++c) a1[c] = E[c];  // the end of the last step's q/m E
    } else {
        pull<MAG>(qm, E, B, S.v, a1);
    }
    const double acc2 = a1[0] * a1[0] + a1[1] * a1[1] + a1[2] * a1[2];
    double dt = S.dt0;
    if (FORM == kSpeculated) {
        limited = !((acc2 * S.hloc) * S.hloc < (4.0 - 4e-9) * (S.speed2 * S.speed2)) || !(dt > 0.0);
    } else {
        const double accel = sqrt(acc2);
        if (accel > 0.0) {
            const double d2 = sqrt(2.0 * S.hloc / accel);
            if (dt < 0.0 || d2 < dt) dt = d2;
        }
        if (dt < 0.0) dt = S.hloc;
        limited = false;
    }
    dt = G.fraction * dt;
    const double hdt = 0.5 * dt;
    double *y = T.x, *w = T.v;
    Place Wq;
    if (INTEG != 0) {
        // half a kick, the drift, the field there and the other half
        double k[3];
        if (MAG) {
#pragma unroll
            for (int c = 0; c < 3; ++c) k[c] = S.v[c];
            kick(num, k, E, B, hdt, qm);
#pragma unroll
            for (int c = 0; c < 3; ++c) y[c] = S.x[c] + dt * k[c];
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) k[c] = S.v[c] + hdt * a1[c];
            const double gk = inv_gamma<GENERAL>(num, k[0], k[1], k[2], inv_c2);
#pragma unroll
            for (int c = 0; c < 3; ++c) y[c] = S.x[c] + dt * gk * k[c];
        }
        locate<CYL, GENERAL>(num, a, G, y, S.at.cell, T.at);
        fields_at<CYL, GENERAL, MAG>(num, a, mag, G, y, T.at, E, B);
        if (MAG) {
            kick(num, k, E, B, hdt, qm);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                w[c] = k[c];
                T.e[c] = E[c];
                T.b[c] = B[c];
            }
        } else {
            double g[3];
            pull<false>(qm, E, B, k, g);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                w[c] = k[c] + hdt * g[c];
                T.e[c] = g[c];
            }
        }
        T.have = true;
    } else {
        double q[3], k2[3], k3[3], k4[3], g[3], sx[3], sv[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sx[c] = gv * S.v[c];
            sv[c] = a1[c];
            q[c] = S.x[c] + hdt * gv * S.v[c];
            k2[c] = S.v[c] + hdt * a1[c];
        }
        const double g2 = inv_gamma<GENERAL>(num, k2[0], k2[1], k2[2], inv_c2);
        locate<CYL, GENERAL>(num, a, G, q, S.at.cell, Wq);
        fields_at<CYL, GENERAL, MAG>(num, a, mag, G, q, Wq, E, B);
        pull<MAG>(qm, E, B, k2, g);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sx[c] = sx[c] + 2.0 * g2 * k2[c];
            sv[c] = sv[c] + 2.0 * g[c];
            q[c] = S.x[c] + hdt * g2 * k2[c];
            k3[c] = S.v[c] + hdt * g[c];
        }
        const double g3 = inv_gamma<GENERAL>(num, k3[0], k3[1], k3[2], inv_c2);
        locate<CYL, GENERAL>(num, a, G, q, S.at.cell, Wq);
        fields_at<CYL, GENERAL, MAG>(num, a, mag, G, q, Wq, E, B);
        pull<MAG>(qm, E, B, k3, g);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sx[c] = sx[c] + 2.0 * g3 * k3[c];
            sv[c] = sv[c] + 2.0 * g[c];
            q[c] = S.x[c] + dt * g3 * k3[c];
            k4[c] = S.v[c] + dt * g[c];
        }
        const double g4 = inv_gamma<GENERAL>(num, k4[0], k4[1], k4[2], inv_c2);
        locate<CYL, GENERAL>(num, a, G, q, S.at.cell, Wq);
        fields_at<CYL, GENERAL, MAG>(num, a, mag, G, q, Wq, E, B);
        pull<MAG>(qm, E, B, k4, g);
        const double dt6 = num.known(dt, 6.0, 1.0 / 6.0);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            y[c] = S.x[c] + dt6 * (sx[c] + g4 * k4[c]);
            w[c] = S.v[c] + dt6 * (sv[c] + g[c]);
        }
        T.have = false;
        locate<CYL, GENERAL>(num, a, G, y, S.at.cell, T.at);
    }
    const double gw = T.gv = inv_gamma<GENERAL>(num, w[0], w[1], w[2], inv_c2);
    set_pace<GENERAL, MAG>(num, a, G, T);

    // the deposit of the step's Hermite midpoint (:372-423); a / 8 is a * 0.125 exactly
    double m0 = 0.5 * (S.x[0] + y[0]) + dt * (gv * S.v[0] - gw * w[0]) * 0.125;
    double m1 = 0.5 * (S.x[1] + y[1]) + dt * (gv * S.v[1] - gw * w[1]) * 0.125;
    const double m2 = 0.5 * (S.x[2] + y[2]) + dt * (gv * S.v[2] - gw * w[2]) * 0.125;
    if (CYL == 1)
        m1 = num.root(m1 * m1 + m2 * m2);
    else if (CYL == 2)
        m1 = G.oy + fabs(m1 - G.oy);
    int cell;
    m0 = uniform_x<GENERAL>(num, a, G, m0, S.at.cell, cell);
    const bool one = !GENERAL || G.P == 1;
    const PatchGeom g = one ? G.base : patch_geom(a, finest_patch(a, G.P, m0, m1));
    const double rphh = one ? g.rphh : 0.0;
    // quotients by the patch's spacing
    num.not_tiny(m0);
    if (CYL != 1) num.not_tiny(m1);
    auto cells_of = [&](double v) {
        return one ? num.known_sound(v, g.phh, rphh) : num.div(v, g.phh);
    };
    const int pnx = (int)g.pnx, pny = (int)g.pny;
    int i = __double2int_rd(cells_of(m0 - g.pox));
    int j = __double2int_rd(cells_of(m1 - g.poy));
    double u = cells_of(m0 - (g.pox + g.phh * (double)i));
    double wr;
    if (CYL == 1) {
        const double low = g.poy + g.phh * (double)j;
        const double high = low + g.phh;
        const double span = high * high - low * low, part = m1 * m1 - low * low;
        wr = one ? num.div_sound(part, span) : num.div(part, span);
    } else {
        wr = cells_of(m1 - (g.poy + g.phh * (double)j));
    }
    if (i < 0) {
        u = 0.0;
        i = 0;
    } else if (i >= pnx - 1) {
        u = 1.0;
        i = pnx - 2;
    }
    if (j < 0) {
        wr = 0.0;
        j = 0;
    } else if (j >= pny - 1) {
        wr = 1.0;
        j = pny - 2;
    }
    D.key = (uint32_t)(g.ofn + (i64)i * pny + j);
    const double ch = G.dq * dt;
    D.c00 = (1.0 - u) * (1.0 - wr) * ch;
    D.c01 = (1.0 - u) * wr * ch;
    D.c10 = u * (1.0 - wr) * ch;
    D.c11 = u * wr * ch;
    // (an intermediate value out of range leaves the end state, or its root, out of range)
    num.not_huge(y[0]);
    if (CYL != 1) num.not_huge(y[1]);
    return !num.odd();
}

// The same with IEEE operations, out of line: for the steps the straight-line form refuses.
template <int CYL, int INTEG, bool GENERAL, bool MAG>
__device__ __noinline__ void advance_plain(const bt_trace_args &a, const bt_magnetic &mag,
                                           const Geo &G, const State &S, State &T, Share &D) {
    bool limited;
    advance<CYL, INTEG, GENERAL, MAG, kIeee>(a, mag, G, S, T, D, limited);
    // (the root's reciprocal, for the straight-line quotients by the radius)
    T.at.y = T.at.r > 0.0 ? 1.0 / T.at.r : 0.0;
}

// The straight-line step with the time that the acceleration sets, out of line: for the steps
// that it limits.
template <int CYL, int INTEG, bool GENERAL, bool MAG>
__device__ __noinline__ bool advance_timed(const bt_trace_args &a, const bt_magnetic &mag,
                                           const Geo &G, const State &S, State &T, Share &D) {
    bool limited;
    return advance<CYL, INTEG, GENERAL, MAG, kTimed>(a, mag, G, S, T, D, limited);
}

// The place and pace of a state whose position and velocity are set.
template <int CYL, bool GENERAL, bool MAG>
__device__ __noinline__ void begin_plain(const bt_trace_args &a, const Geo &G, State &S) {
    Num<false> num;
    S.gv = inv_gamma<GENERAL>(num, S.v[0], S.v[1], S.v[2], G.inv_c2);
    locate<CYL, GENERAL>(num, a, G, S.x, S.at.cell, S.at);
    // (the root's reciprocal, for the straight-line quotients by the radius)
    S.at.y = S.at.r > 0.0 ? 1.0 / S.at.r : 0.0;
    set_pace<GENERAL, MAG>(num, a, G, S);
}

// The kernel is specialised on the geometry (0 planar, 1 cylindrical, 2 symmetry plane),
// the integrator (0 RK4, 1 Boris) and GENERAL: refined patches, a graded x axis or
// relativity.  Without them the mesh is one patch, whose shape is read once, and gamma is
// exactly 1; the operations on every value are the general kernel's, so the results are.
// MAG: the reference's NumPy tracer's step in a magnetic field instead (tracer.py:851-1054):
// q/m (E + v x B) at every stage, Boris with the rotation, and every step that ends in a
// cell touching an electrode pauses (status -2) for the caller's exact inside test.
//
// The live trajectories are act[0, *live); the grid covers `stride` >= *live threads, the
// live count when the host last read it, and the records of step s of thread m go to slot
// s * stride + m.  Threads past the live count fill their slots with the sentinel.  A
// window with live trajectories sets *records_end to `end`, the end of its slots, so the
// deposit sorts no window that had none.
//
// One thread's window (m < stride): whether its trajectory is still live afterwards.
template <int CYL, int INTEG, bool GENERAL, bool MAG, bool BATCH>
__device__ __forceinline__ bool trace_thread(const Trace &tr, const i64 *__restrict__ act,
                                             i64 m, i64 n_act, i64 stride, int S,
                                             uint32_t *__restrict__ keys,
                                             DepositRec *__restrict__ rec, uint32_t sentinel) {
    if (m >= n_act) {
        for (int s = 0; s < S; ++s) keys[(i64)s * stride + m] = sentinel;
        return false;
    }
    const bt_trace_args &a = tr.a;
    const i64 k = act[m];
    // the one patch of a non-general mesh (of the trajectory's candidate in a batch)
    const i64 cand = BATCH ? (i64)__ldg(tr.cand + k) : 0;
    Geo G;
    G.P = GENERAL ? (int)a.n_patches : 1;
    G.base = patch_geom(a, cand);
    G.base.rphh = known_reciprocal(G.base.phh);
    const i64 nx = BATCH ? G.base.pnx : tr.nx, ny = BATCH ? G.base.pny : tr.ny;
    G.ox = BATCH ? G.base.pox : a.origin_x;
    G.oy = BATCH ? G.base.poy : a.origin_y;
    G.h = BATCH ? G.base.phh : a.h;
    G.rh = BATCH ? G.base.rphh : known_reciprocal(a.h);
    G.rhz = MAG ? known_reciprocal(tr.mag.hz) : 1.0;
    G.qm = a.qm[k];
    G.dq = a.dq[k];
    G.fraction = a.step_fraction;
    G.inv_c2 = a.inv_c2;
    G.graded = GENERAL && a.graded != 0;
    G.n_x_nodes = (int)a.n_x_nodes;
    G.same = G.P == 1 && G.base.pox == G.ox && G.base.poy == G.oy && G.base.phh == G.h;
    G.fast = G.rh != 0.0 && G.base.rphh != 0.0 && G.rhz != 0.0 && (GENERAL || G.same) &&
             sound_origin(G.ox) && sound_origin(G.oy) && sound_origin(G.base.pox) &&
             sound_origin(G.base.poy);
    const double upper_x = BATCH ? __ldg(a.patch_real + cand * 7 + 5) : a.upper_x;
    const double upper_y = BATCH ? __ldg(a.patch_real + cand * 7 + 6) : a.upper_y;
    const i64 *__restrict__ cells = BATCH ? a.cells + __ldg(tr.cell_off + cand) : a.cells;
    const i64 n = a.n;
    State now;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        now.x[c] = a.x[c * n + k];
        now.v[c] = a.v[c * n + k];
        now.e[c] = now.b[c] = 0.0;
    }
    now.have = false;
    now.at.cell = G.graded ? first_cell(now.x[0], a.x_nodes, G.n_x_nodes) : 0;
    {
        State first = now;
        const Geo g = G;
        begin_plain<CYL, GENERAL, MAG>(a, g, first);
        now = first;
    }
    const i64 slot = a.path_slot[k];
    i64 ns = a.steps[k];
    i64 st = -1;
    // the first planes in registers: a step's crossing test is two comparisons a plane
    constexpr int kHeldPlanes = 2;
    double held[kHeldPlanes];
#pragma unroll
    for (int p = 0; p < kHeldPlanes; ++p)
        held[p] = p < a.n_planes ? a.planes[p] : __longlong_as_double(0x7ff8000000000000LL);
    // The records of consecutive steps in one cell are summed into one (the run's): it goes
    // to the slot of the run's last step, the slots of its other steps hold the sentinel.
    i64 run_slot = -1;
    uint32_t run_key = sentinel;
    double r00 = 0.0, r01 = 0.0, r10 = 0.0, r11 = 0.0;
    // a point below the mesh (only a malformed geometry puts one there) takes its first cell,
    // where the reference indexes outside the table
    auto last_cell = [](double u, i64 nodes) {
        return max(min(__double2int_rz(u), (int)nodes - 2), 0);
    };
    auto cell_at = [&](const Place &W) {
        return __ldg(cells + (i64)last_cell(W.sx, nx) * (ny - 1) + last_cell(W.sy, ny));
    };
    int s = 0;
    for (; s < S; ++s) {
        if (ns >= a.max_steps) break;
        State next;
        Share D;
        bool limited;
        const bool ok =
            advance<CYL, INTEG, GENERAL, MAG, kSpeculated>(a, tr.mag, G, now, next, D, limited) &&
            G.fast;
        // the end's cell in the electrode table: asked for here, where the lookup runs beside
        // the rest of the step's arithmetic
        i64 cell = cell_at(next.at);
        if (!ok || limited) {
            // copies, so that only this branch keeps anything in memory
            const State from = now;
            const Geo g = G;
            State to;
            Share d;
            if (!ok || !advance_timed<CYL, INTEG, GENERAL, MAG>(a, tr.mag, g, from, to, d))
                advance_plain<CYL, INTEG, GENERAL, MAG>(a, tr.mag, g, from, to, d);
            next = to;
            D = d;
            cell = cell_at(next.at);
        }
        if (run_slot >= 0 && D.key == run_key) {
            // the step stays in the run's cell: its charge joins the run's record
            keys[run_slot] = sentinel;
            r00 = r00 + D.c00;
            r01 = r01 + D.c01;
            r10 = r10 + D.c10;
            r11 = r11 + D.c11;
        } else {
            if (run_slot >= 0) {
                keys[run_slot] = run_key;
                rec[run_slot] = DepositRec{r00, r01, r10, r11};
            }
            run_key = D.key;
            r00 = D.c00;
            r01 = D.c01;
            r10 = D.c10;
            r11 = D.c11;
        }
        run_slot = (i64)s * stride + m;
        ns = ns + 1;

        bool crossing = a.n_planes > kHeldPlanes;
#pragma unroll
        for (int p = 0; p < kHeldPlanes; ++p)
            crossing |= (now.x[0] < held[p]) != (next.x[0] < held[p]);
        if (crossing) {
            for (i64 p = 0; p < a.n_planes; ++p) {
                const double xp = a.planes[p];
                const double before = now.x[0] - xp;
                const double after = next.x[0] - xp;
                if ((before < 0.0) != (after < 0.0)) {
                    const double sc = before / (before - after);
                    i64 *cnt = a.counts + k * a.n_planes + p;
                    const i64 c = *cnt;
                    if (c < a.capacity) {
                        double *hit = a.hits + ((k * a.n_planes + p) * a.capacity + c) * 8;
                        const double gv = GENERAL ? now.gv : 1.0;
                        const double gw = GENERAL ? next.gv : 1.0;
                        hit[0] = xp;
                        hit[1] = now.x[1] + sc * (next.x[1] - now.x[1]);
                        hit[2] = now.x[2] + sc * (next.x[2] - now.x[2]);
                        hit[3] = gv * now.v[0] + sc * (gw * next.v[0] - gv * now.v[0]);
                        hit[4] = gv * now.v[1] + sc * (gw * next.v[1] - gv * now.v[1]);
                        hit[5] = gv * now.v[2] + sc * (gw * next.v[2] - gv * now.v[2]);
                        hit[6] = after >= 0.0 ? 1.0 : -1.0;
                        hit[7] = 1.0 * (double)ns;
                    }
                    *cnt = c + 1;
                }
            }
        }
        now = next;

        const double px = now.at.lx, py = now.at.r;
        if (slot >= 0) {
            const i64 c = a.path_count[slot];
            if (c < a.path_capacity) {
                a.paths[(slot * a.path_capacity + c) * 2 + 0] = now.x[0];
                a.paths[(slot * a.path_capacity + c) * 2 + 1] = py;
            }
            a.path_count[slot] = c + 1;
        }
        if (px >= upper_x) {
            st = 0;
        } else if (px < G.ox) {
            st = 1;
        } else if (py > upper_y || (CYL == 0 && py < G.oy)) {
            st = 2;
        } else {
            const double ux = now.at.sx, uy = now.at.sy;
            if (MAG && cell >= 0) {
                st = -2;  // the caller tests the electrodes' shapes
            } else if (cell >= 0) {
                const int i = last_cell(ux, nx), j = last_cell(uy, ny);
                const i64 R = a.refine;
                i64 si = (i64)((ux - (double)i) * (double)R);
                if (si < 0)
                    si = 0;
                else if (si > R - 1)
                    si = R - 1;
                i64 sj = (i64)((uy - (double)j) * (double)R);
                if (sj < 0)
                    sj = 0;
                else if (sj > R - 1)
                    sj = R - 1;
                const i64 e = __ldg(a.subcells + (cell * R + si) * R + sj);
                if (e >= 0) {
                    st = 3;
                    a.electrode[k] = e;
                } else if (e == -2 && BATCH && tr.shape_first) {
                    // the candidate's own electrodes, tested here at the point's mesh
                    // coordinates: the caller's test of a paused trajectory
                    const i64 s0 = __ldg(tr.shape_first + cand);
                    const Shapes sh{__ldg(tr.shape_first + cand + 1) - s0, tr.shapes.kind + s0,
                                    tr.shapes.offset + s0, tr.shapes.params};
                    const i64 hit = inside_solid(sh, px, py);
                    if (hit >= 0) {
                        st = 3;
                        a.electrode[k] = hit;
                    }
                } else if (e == -2) {
                    st = -2;
                }
            }
        }
        if (st != -1) {
            ++s;
            break;
        }
    }
    if (run_slot >= 0) {
        keys[run_slot] = run_key;
        rec[run_slot] = DepositRec{r00, r01, r10, r11};
    }
    // the slots of the steps not taken hold no record
    for (; s < S; ++s) keys[(i64)s * stride + m] = sentinel;
    if (st == -1 && ns >= a.max_steps) st = 4;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        a.x[c * n + k] = now.x[c];
        a.v[c * n + k] = now.v[c];
    }
    a.steps[k] = ns;
    a.status[k] = st;
    return st == -1;
}

// The window: every thread's trajectory, then each block's count of live trajectories and
// every thread's flag, for compact_live.  BATCH: the trajectories of many candidate meshes
// in one launch (Trace::cand).  BLOCKS: the blocks an SM is to hold, which bounds a thread's
// registers (255 for two, 168 for three; see trace_all for which is launched).
template <int CYL, int INTEG, bool GENERAL, bool MAG, bool BATCH, int BLOCKS>
__global__ void __launch_bounds__(128, BLOCKS)
    trace_window(const __grid_constant__ Trace tr, const i64 *__restrict__ act, const i64 *__restrict__ live, i64 stride,
                 int S, uint32_t *__restrict__ keys, DepositRec *__restrict__ rec,
                 uint32_t sentinel, i64 *__restrict__ records_end, i64 end,
                 uint32_t *__restrict__ block_live, uint8_t *__restrict__ alive) {
    const i64 m = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const i64 n_act = *live;
    if (m == 0 && n_act > 0) *records_end = end;
    bool still = false;
    if (m < stride)
        still = trace_thread<CYL, INTEG, GENERAL, MAG, BATCH>(tr, act, m, n_act, stride, S, keys,
                                                              rec, sentinel);
    const int count = __syncthreads_count(still);
    if (m < stride) alive[m] = still ? 1 : 0;
    if (threadIdx.x == 0) block_live[blockIdx.x] = (uint32_t)count;
}

// -- order-preserving compaction of the live trajectories ----------------------------------

// Windows of more blocks than this have their blocks' offsets scanned by block_offsets
// (each compact_live block would otherwise add up all the counts before its own).
constexpr int kSumBlocks = 2048;

// offsets[b] = the live trajectories of the window's blocks before b (one block, in chunks
// of 1024).
__global__ void __launch_bounds__(1024) block_offsets(const uint32_t *__restrict__ block_live,
                                                      int nblocks, uint32_t *__restrict__ offsets) {
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t carry;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) carry = 0;
    __syncthreads();
    for (int start = 0; start < nblocks; start += 1024) {
        const int b = start + t;
        const uint32_t v = b < nblocks ? block_live[b] : 0u;
        uint32_t x = v;
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
            if (lane >= off) x += y;
        }
        if (lane == 31) warp_sums[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint32_t w = warp_sums[lane];
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, w, off);
                if (lane >= off) w += y;
            }
            warp_sums[lane] = w;
        }
        __syncthreads();
        const uint32_t inclusive = x + (warp > 0 ? warp_sums[warp - 1] : 0u) + carry;
        if (b < nblocks) offsets[b] = inclusive - v;
        __syncthreads();
        if (t == 1023) carry = inclusive;
        __syncthreads();
    }
}

// act_out = the live trajectories of act, in order, and *live_out their count, from a
// window's per-block counts and flags (the window's grid of 128-thread blocks); `offsets`,
// when not NULL, holds each block's count of the live trajectories before it.
__global__ void __launch_bounds__(128) compact_live(const i64 *__restrict__ act,
                                                    const uint8_t *__restrict__ alive,
                                                    const uint32_t *__restrict__ block_live,
                                                    const uint32_t *__restrict__ offsets,
                                                    i64 stride, i64 *__restrict__ act_out,
                                                    i64 *__restrict__ live_out) {
    __shared__ uint32_t part[4], warp_first[4];
    const int b = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t before = 0;  // the live trajectories of the blocks before this one
    if (offsets)
        before = t == 0 ? offsets[b] : 0u;
    else
        for (int q = t; q < b; q += 128) before += block_live[q];
    for (int off = 16; off > 0; off >>= 1) before += __shfl_down_sync(0xffffffffu, before, off);
    if (lane == 0) part[warp] = before;
    const i64 m = (i64)b * 128 + t;
    const bool a = m < stride && alive[m] != 0;
    const unsigned ballot = __ballot_sync(0xffffffffu, a);
    if (lane == 0) warp_first[warp] = __popc(ballot);
    __syncthreads();
    const uint32_t offset = part[0] + part[1] + part[2] + part[3];
    uint32_t rank = offset;
    for (int w = 0; w < warp; ++w) rank += warp_first[w];
    rank += __popc(ballot & ((1u << lane) - 1u));
    if (a) act_out[rank] = act[m];
    if (b == (int)gridDim.x - 1 && t == 0) *live_out = offset + block_live[b];
}

__global__ void set_count(i64 *__restrict__ count, i64 value) { *count = value; }

}  // namespace

}  // namespace bt

namespace bt {
namespace {

// Windows launched between two reads of the live count.
constexpr int kGroup = 4;

// Record slots per deposit batch, at most: a batch is a group's windows when they hold
// fewer.  A batch is deposited at the end of its group, under the next group's windows,
// so only the last group's deposit is left when the trace ends.
constexpr int64_t kBatchRecords = (int64_t)1 << 24;

// Points the context's launches at `side` for its lifetime.
struct SideStream {
    bt_ctx *ctx;
    cudaStream_t saved;
    SideStream(bt_ctx *c, cudaStream_t side) : ctx(c), saved(c->stream) { ctx->stream = side; }
    ~SideStream() { ctx->stream = saved; }
};

// Windows between reads of the live count for a batch: as many as keep a group's record
// slots within kBatchGroupRecords (at least one, at most kGroup).
constexpr int64_t kBatchGroupRecords = (int64_t)1 << 26;

void trace_all(bt_ctx *ctx, const bt_trace_args *args, const bt_magnetic *mag, int64_t window,
               const bt_trace_batch *batch = nullptr) {
    {
        BT_REQUIRE(ctx && args, "trace: null argument");
        const bt_trace_args &a = *args;
        BT_REQUIRE(a.n_patches >= 1 && a.patch_int && a.patch_real, "trace: no patches");
        BT_REQUIRE(a.n_active >= 0 && a.n >= 0, "trace: negative sizes");
        BT_REQUIRE(a.capacity >= 0 && a.path_capacity >= 0 && a.n_planes >= 0,
                   "trace: negative buffer sizes");
        BT_REQUIRE(a.refine >= 1, "trace: refine must be positive");
        BT_REQUIRE(!a.graded || a.n_x_nodes >= 2, "trace: a graded axis needs its nodes");
        BT_REQUIRE(a.n_nodes < (int64_t)0xffffffffLL, "trace: too many nodes for 32-bit keys");
        bt::Trace tr;
        tr.a = a;
        tr.mag = mag ? *mag : bt_magnetic{};
        if (mag) {
            BT_REQUIRE(mag->mode == 1 || mag->mode == 2, "trace: magnetic mode must be 1 or 2");
            BT_REQUIRE(mag->order >= 0 && mag->order <= 6, "trace: magnetic order must be 0 to 6");
            BT_REQUIRE(mag->n >= 8 && mag->samples, "trace: the profile needs 8 samples");
            BT_REQUIRE(mag->hz > 0.0, "trace: the profile spacing must be positive");
            BT_REQUIRE((mag->mode == 1) == (a.cylindrical == 1),
                       "trace: mode 1 needs a cylindrical mesh, mode 2 a planar one");
            BT_REQUIRE(a.inv_c2 == 0.0 && a.n_patches == 1,
                       "trace: the magnetic trace is non-relativistic on one patch");
            BT_REQUIRE(a.cylindrical != 2, "trace: no magnetic field with a symmetry plane");
        }
        tr.cand = nullptr;
        tr.cell_off = nullptr;
        tr.shape_first = nullptr;
        tr.shapes = bt::Shapes{0, nullptr, nullptr, nullptr};
        if (batch) {
            // every candidate's one patch: shapes of at least 2 x 2 nodes whose node ranges
            // tile [0, n_nodes) in order (the deposit finds a node's candidate by bisection)
            BT_REQUIRE(!mag, "trace: a batch takes no magnetic field");
            BT_REQUIRE(batch->n_candidates >= 1 && batch->n_candidates == a.n_patches,
                       "trace: a batch needs one patch row per candidate");
            BT_REQUIRE(batch->candidate && batch->cell_offset, "trace: null batch table");
            BT_REQUIRE(!a.graded && a.inv_c2 == 0.0,
                       "trace: a batch takes uniform, non-relativistic meshes");
            std::vector<int64_t> rows((size_t)6 * a.n_patches);
            BT_CUDA(cudaMemcpyAsync(rows.data(), a.patch_int, sizeof(int64_t) * rows.size(),
                                    cudaMemcpyDeviceToHost, ctx->stream));
            BT_CUDA(cudaStreamSynchronize(ctx->stream));
            int64_t next = 0;
            for (int64_t c = 0; c < a.n_patches; ++c) {
                const int64_t *r = rows.data() + 6 * c;
                BT_REQUIRE(r[0] >= 2 && r[1] >= 2, "trace: a candidate needs at least 2 x 2 nodes");
                BT_REQUIRE(r[4] == r[0] * r[1] && r[5] == next,
                           "trace: the candidates' nodes must follow one another from 0");
                next += r[4];
            }
            BT_REQUIRE(next == a.n_nodes, "trace: the candidates' nodes must fill n_nodes");
            tr.cand = batch->candidate;
            tr.cell_off = batch->cell_offset;
            if (batch->shape_first) {
                BT_REQUIRE(batch->shape_kind && batch->shape_offset && batch->shape_params,
                           "trace: a batch's shapes need their kind, offset and parameters");
                tr.shape_first = batch->shape_first;
                tr.shapes = bt::Shapes{0, batch->shape_kind, batch->shape_offset,
                                       batch->shape_params};
            }
            tr.nx = tr.ny = 0;
        } else {
            // the last patch's shape, for the exit and electrode tests
            int64_t last[6];
            BT_CUDA(cudaMemcpyAsync(last, a.patch_int + (a.n_patches - 1) * 6, sizeof(last),
                                    cudaMemcpyDeviceToHost, ctx->stream));
            BT_CUDA(cudaStreamSynchronize(ctx->stream));
            tr.nx = last[0];
            tr.ny = last[1];
            BT_REQUIRE(tr.nx >= 2 && tr.ny >= 2, "trace: the mesh needs at least 2 x 2 nodes");
        }
        BT_REQUIRE(a.cylindrical >= 0 && a.cylindrical <= 2, "trace: geometry must be 0, 1 or 2");
        const int S = window > 0 ? (int)window : 64;
        const bool general = !batch && (a.n_patches > 1 || a.graded != 0 || a.inv_c2 != 0.0);
        ctx->last_windows = ctx->last_records = ctx->last_flushes = 0;
        if (a.n_active == 0) return;
        bt::TraceScratch &ts = ctx->trace;
        cudaStream_t st = ctx->stream;
        const uint32_t sentinel = (uint32_t)a.n_nodes;
        // Two record buffers: the windows fill one while the records of the other are sorted
        // and reduced into charge[0] on the side stream, in the order the buffers were
        // filled, so the deposit runs under the next windows and the sums are the same
        // whatever the timing.  A buffer is deposited at the end of the group that brought
        // it to `flush_at` records (or on filling up within a group).  A batch's windows
        // are large: its groups hold fewer of them, so the buffers stay within a few GB.
        const int64_t per_window = a.n_active * (int64_t)S;
        int group = kGroup;
        if (batch) {
            const int64_t fit = std::max<int64_t>(1, kBatchGroupRecords / std::max<int64_t>(per_window, 1));
            group = (int)std::min<int64_t>(batch->group > 0 ? batch->group : fit, kGroup);
        }
        const int64_t flush_at = std::min<int64_t>(kBatchRecords, group * per_window);
        const int64_t capacity = flush_at + group * per_window;
        uint32_t *keys[2];
        bt::DepositRec *rec[2];
        for (int b = 0; b < 2; ++b) {
            keys[b] = ts.rec_keys[b].as<uint32_t>(capacity);
            rec[b] = ts.rec[b].as<bt::DepositRec>(capacity);
        }
        if (!ts.side) {
            BT_CUDA(cudaStreamCreateWithFlags(&ts.side, cudaStreamNonBlocking));
            for (int b = 0; b < 2; ++b) {
                BT_CUDA(cudaEventCreateWithFlags(&ts.filled[b], cudaEventDisableTiming));
                BT_CUDA(cudaEventCreateWithFlags(&ts.drained[b], cudaEventDisableTiming));
            }
        }
        int64_t *act_a = ts.active_a.as<int64_t>(a.n_active);
        int64_t *act_b = ts.active_b.as<int64_t>(a.n_active);
        // the window's per-block live counts, and room after them for their offsets
        uint32_t *block_live =
            ts.block_counts.as<uint32_t>(2 * (size_t)bt::blocks_for(a.n_active, 128));
        uint8_t *alive = ts.alive.as<uint8_t>(a.n_active);
        // live[2]: the live count before and after a window's compaction; records_end[2]:
        // where the slots of each buffer's last window with live trajectories end
        int64_t *live = ts.n_alive.as<int64_t>(4);
        int64_t *records_end = live + 2;
        int64_t *n_alive_host = static_cast<int64_t *>(ctx->host.get(sizeof(int64_t)));
        BT_CUDA(cudaMemcpyAsync(act_a, a.active, sizeof(int64_t) * a.n_active,
                                cudaMemcpyDeviceToDevice, st));
        BT_CUDA(cudaMemsetAsync(records_end, 0, 2 * sizeof(int64_t), st));
        BT_LAUNCH(ctx, bt::set_count, 1, 1, 0, st, live, a.n_active);
        // A batch's deposits add their per-cell sums up over the whole trace and reach the
        // nodes once at its end (a flush then costs only its records, not every node of
        // every candidate).
        if (batch) bt::deposit_cells_reset(ctx, a.n_nodes);
        bt::NodeLayout layout{a.patch_int, a.n_patches, tr.nx, tr.ny, a.n_nodes, batch != nullptr};
        int64_t bound = a.n_active, used = 0;
        int lv = 0;
        int cur = 0;
        bool pending[2] = {false, false};
        // deposit buffer `cur` on the side stream and switch the windows to the other one
        auto flush = [&] {
            if (used == 0) return;
            BT_CUDA(cudaEventRecord(ts.filled[cur], st));
            BT_CUDA(cudaStreamWaitEvent(ts.side, ts.filled[cur], 0));
            {
                SideStream on_side(ctx, ts.side);
                bt::Timed timed(ctx, "deposit");
                bt::deposit_records(ctx, keys[cur], rec[cur], used, records_end + cur, sentinel,
                                    a.charge, layout, batch != nullptr);
            }
            BT_CUDA(cudaMemsetAsync(records_end + cur, 0, sizeof(int64_t), ts.side));
            BT_CUDA(cudaEventRecord(ts.drained[cur], ts.side));
            pending[cur] = true;
            ctx->last_records += used;
            ctx->last_flushes += 1;
            used = 0;
            cur ^= 1;
            if (pending[cur]) BT_CUDA(cudaStreamWaitEvent(st, ts.drained[cur], 0));
        };
        // The windows go in groups of kGroup between reads of the live count: each reads
        // the count on the device, and a window after the last trajectory ended does no work.
        while (bound > 0) {
            for (int g = 0; g < group; ++g) {
                const int64_t need = bound * (int64_t)S;
                if (used + need > capacity) flush();
                unsigned grid = 0;
                {
                    bt::Timed timed(ctx, "trace_window");
                    grid = (unsigned)bt::blocks_for(bound, 128);
                    const int64_t launched = ctx->launch_count;
                    // A window whose blocks fit two a multiprocessor has warps to spare for
                    // none: 255 registers let the lookups' chains run side by side (20,000
                    // rings, 157 blocks: 132 us a window against 159 with 168 registers).
                    // A larger one hides latency with a third block (40,000 rings: 7.3 ms a
                    // trace against 8.3), as do the magnetic trace's (52 ms against 64).  A
                    // batch's windows come down to the first kind as its candidates finish.
                    const bool wide = !mag && grid <= (unsigned)(2 * ctx->num_sms);
#define BT_TRACE_CASE_N(C, I, G, M, B, N)                                                       \
    if (a.cylindrical == C && (a.integrator != 0) == (I != 0) && general == G &&                 \
        (mag != nullptr) == M && (batch != nullptr) == B && wide == (N == 2))                    \
        BT_LAUNCH(ctx, (bt::trace_window<C, I, G, M, B, N>), grid, 128, 0, st, tr, act_a,         \
                  live + lv, bound, S, keys[cur] + used, rec[cur] + used, sentinel,               \
                  records_end + cur, used + need, block_live, alive);
#define BT_TRACE_CASE_B(C, I, G, M, B)                                                          \
    BT_TRACE_CASE_N(C, I, G, M, B, 3) BT_TRACE_CASE_N(C, I, G, M, B, 2)
#define BT_TRACE_CASE(C, I, G, M)                                                               \
    BT_TRACE_CASE_N(C, I, G, M, false, 3)                                                         \
    if (!M) { BT_TRACE_CASE_N(C, I, G, false, false, 2) }
                    BT_TRACE_CASE(0, 0, false, false) BT_TRACE_CASE(0, 0, true, false)
                    BT_TRACE_CASE(0, 1, false, false) BT_TRACE_CASE(0, 1, true, false)
                    BT_TRACE_CASE(1, 0, false, false) BT_TRACE_CASE(1, 0, true, false)
                    BT_TRACE_CASE(1, 1, false, false) BT_TRACE_CASE(1, 1, true, false)
                    BT_TRACE_CASE(2, 0, false, false) BT_TRACE_CASE(2, 0, true, false)
                    BT_TRACE_CASE(2, 1, false, false) BT_TRACE_CASE(2, 1, true, false)
                    BT_TRACE_CASE(0, 0, false, true) BT_TRACE_CASE(0, 0, true, true)
                    BT_TRACE_CASE(0, 1, false, true) BT_TRACE_CASE(0, 1, true, true)
                    BT_TRACE_CASE(1, 0, false, true) BT_TRACE_CASE(1, 0, true, true)
                    BT_TRACE_CASE(1, 1, false, true) BT_TRACE_CASE(1, 1, true, true)
                    BT_TRACE_CASE_B(0, 0, false, false, true) BT_TRACE_CASE_B(0, 1, false, false, true)
                    BT_TRACE_CASE_B(1, 0, false, false, true) BT_TRACE_CASE_B(1, 1, false, false, true)
                    BT_TRACE_CASE_B(2, 0, false, false, true) BT_TRACE_CASE_B(2, 1, false, false, true)
#undef BT_TRACE_CASE
#undef BT_TRACE_CASE_B
#undef BT_TRACE_CASE_N
                    BT_REQUIRE(ctx->launch_count > launched,
                               "trace: no kernel for these settings");
                }
                BT_CHECK_LAUNCH();
                used += need;
                ctx->last_windows += 1;
                uint32_t *offsets = nullptr;
                if (grid > (unsigned)bt::kSumBlocks) {
                    offsets = block_live + grid;
                    BT_LAUNCH(ctx, bt::block_offsets, 1, 1024, 0, st, block_live, (int)grid,
                              offsets);
                }
                BT_LAUNCH(ctx, bt::compact_live, grid, 128, 0, st, act_a, alive, block_live,
                          offsets, bound, act_b, live + (lv ^ 1));
                BT_CHECK_LAUNCH();
                std::swap(act_a, act_b);
                lv ^= 1;
            }
            BT_CUDA(cudaMemcpyAsync(n_alive_host, live + lv, sizeof(int64_t),
                                    cudaMemcpyDeviceToHost, st));
            BT_CUDA(cudaStreamSynchronize(st));
            bound = *n_alive_host;
            if (used >= flush_at) flush();
        }
        flush();
        // the caller's stream continues once every deposit is in charge[0]
        for (int b = 0; b < 2; ++b)
            if (pending[b]) BT_CUDA(cudaStreamWaitEvent(st, ts.drained[b], 0));
        if (batch) bt::deposit_cells_finish(ctx, a.charge, layout);
    }
}

}  // namespace
}  // namespace bt

// trace_fast.cu compiles this file again with contracted multiply-adds; its entry points
// carry the suffix _fast.
#ifdef BT_TRACE_FAST
#define BT_TRACE_ENTRY(name) name##_fast
#else
#define BT_TRACE_ENTRY(name) name
#endif

extern "C" int BT_TRACE_ENTRY(bt_trace_trajectories_2d)(bt_ctx *ctx, const bt_trace_args *args,
                                                        int64_t window) {
    return bt::guarded([&] { bt::trace_all(ctx, args, nullptr, window); });
}

extern "C" int BT_TRACE_ENTRY(bt_trace_trajectories_2d_magnetic)(bt_ctx *ctx,
                                                                 const bt_trace_args *args,
                                                                 const bt_magnetic *magnetic,
                                                                 int64_t window) {
    return bt::guarded([&] {
        BT_REQUIRE(magnetic, "trace: null magnetic field");
        bt::trace_all(ctx, args, magnetic, window);
    });
}

extern "C" int BT_TRACE_ENTRY(bt_trace_trajectories_2d_batch)(bt_ctx *ctx,
                                                              const bt_trace_args *args,
                                                              const bt_trace_batch *batch,
                                                              int64_t window) {
    return bt::guarded([&] {
        BT_REQUIRE(batch, "trace: null batch");
        bt::trace_all(ctx, args, nullptr, window, batch);
    });
}

#ifndef BT_TRACE_FAST
extern "C" int bt_trace_last_stats(bt_ctx *ctx, int64_t *windows, int64_t *records,
                                   int64_t *deposit_flushes) {
    return bt::guarded([&] {
        BT_REQUIRE(ctx, "trace stats: null context");
        if (windows) *windows = ctx->last_windows;
        if (records) *records = ctx->last_records;
        if (deposit_flushes) *deposit_flushes = ctx->last_flushes;
    });
}
#endif
