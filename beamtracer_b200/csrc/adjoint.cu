// The adjoint of the trace: the reverse of trace.cu's RK4 step for the differentiation form
// of the design workload (planar or cylindrical, RK4, one uniform patch, no magnetic
// field, not relativistic).  No counterpart in the reference, which differentiates by
// finite differences of whole solves.
//
// The trace maps the edge fields (fx, fy) to the node charges it deposits and the plane
// crossings it records.  Given the adjoints of those outputs -- charge_seed on the nodes,
// hit_seed on the crossings' points and velocities -- the sweep accumulates the adjoint
// of the edge fields: every gather of the field at a stage point is reversed into a
// scatter onto the same four edges with the same bilinear weights, so gather and deposit
// are each other's transposes.
//
// One thread per trajectory.  A first pass replays every trajectory for the steps it took
// in the forward trace and keeps its state every kSegment steps (checkpoints, the memory
// bound: 6 doubles a trajectory every 64 steps).  The sweep walks the segments from the
// last: it replays a segment's steps from its checkpoint into local memory, then reverses
// them one by one (each step recomputed from its start state), carrying the adjoint of the
// trajectory's state backwards.  The replay is the trace's step, term by term, in the same
// order and with the same roundings (--fmad=false), so it visits the same states bit for
// bit.  The non-smooth parts of the step are taken as they fell in the forward trace: the
// branch of the step size's minimum, the cells of every lookup, the crossings, the clamps
// of the deposit at the mesh's edges.  The scatter adds each run of gathers in one cell in
// registers and the runs' sums to the edges by atomic additions (their order varies from
// run to run, so the adjoint is reproducible to rounding, not bit for bit).
#include "common.cuh"

namespace bt {
namespace {

constexpr int kSegment = 64;   // steps between checkpoints
constexpr int kMaxPlanes = 8;  // plane crossings the sweep follows
// One warp a block: a solve's few thousand trajectories spread over every SM (128-thread
// blocks left most of the 148 SMs idle on 8,000 trajectories).
constexpr int kAdjThreads = 32;

struct Grid {
    const double *fx, *fy;
    int nx, ny;
    double ox, oy, h, rh;
    double ih;  // 1 / h
};

__device__ __forceinline__ int clamp_cell(int i, int lo, int hi) { return min(max(i, lo), hi); }

// A field evaluation at a stage point, with what its reverse needs: the lookups' cells and
// weights (of E_x and E_y, trace.cu's edge_field_cells, the same expressions), E_y, the
// derivatives of the two along the weights, the radius' reciprocal and unit vector.
struct Stage {
    int ix, jx, iy, jy;
    double ux, wx, uy, wy;
    double ey;
    double dex_du, dex_dw, dey_du, dey_dw;
    double cy, cz, ir;
};

// q/m E at a point, as trace.cu forms it (the radius and its unit vector in cylindrical
// geometry).  Num<true>: straight-line roots and quotients (common.cuh), and the cells of
// s + 1/2 from those of s, as the trace's own step.
template <int CYL, class N>
__device__ __forceinline__ void accel(N &num, const Grid &G, double qm, const double *q, double *a,
                                      Stage &g) {
    double qy = q[1];
    g.cy = g.cz = g.ir = 0.0;
    if (CYL == 1) {
        double y;
        qy = num.root(q[1] * q[1] + q[2] * q[2], y);
        const bool off_axis = qy > 0.0;
        const double ir = N::fast ? num.inverse(qy, y) : 1.0 / qy;
        const double uy = num.over(q[1], qy, ir), uz = num.over(q[2], qy, ir);
        g.cy = off_axis ? uy : 0.0;
        g.cz = off_axis ? uz : 0.0;
        g.ir = off_axis ? ir : 0.0;
    }
    // (the coordinates tested, not their differences from the origin; a radius is its root's)
    num.not_tiny(q[0]);
    if (CYL != 1) num.not_tiny(qy);
    const double sx = num.known_sound(q[0] - G.ox, G.h, G.rh);
    const double sy = num.known_sound(qy - G.oy, G.h, G.rh);
    const double hx = sx + 0.5, hy = sy + 0.5;
    if (N::fast) {
        const int i = __double2int_rd(sx), j = __double2int_rd(sy);
        const double fi = (double)i, fj = (double)j;
        const bool up_i = hx >= fi + 1.0, up_j = hy >= fj + 1.0;
        g.ix = clamp_cell(clamp_cell(i, -1, G.nx - 1) + (up_i ? 1 : 0), 0, G.nx - 1);
        g.jx = clamp_cell(j, 0, G.ny - 2);
        g.iy = clamp_cell(i, 0, G.nx - 2);
        g.jy = clamp_cell(clamp_cell(j, -1, G.ny - 1) + (up_j ? 1 : 0), 0, G.ny - 1);
        g.uy = sx - fi;
        g.wx = sy - fj;
        g.ux = hx - (up_i ? fi + 1.0 : fi);
        g.wy = hy - (up_j ? fj + 1.0 : fj);
        if (g.iy != i || g.jx != j) {  // past the mesh's edge
            g.ux = hx - (double)g.ix;
            g.wx = sy - (double)g.jx;
            g.uy = sx - (double)g.iy;
            g.wy = hy - (double)g.jy;
        }
    } else {
        g.ix = clamp_cell(__double2int_rd(hx), 0, G.nx - 1);
        g.jx = clamp_cell(__double2int_rd(sy), 0, G.ny - 2);
        g.iy = clamp_cell(__double2int_rd(sx), 0, G.nx - 2);
        g.jy = clamp_cell(__double2int_rd(hy), 0, G.ny - 1);
        g.ux = hx - (double)g.ix;
        g.wx = sy - (double)g.jx;
        g.uy = sx - (double)g.iy;
        g.wy = hy - (double)g.jy;
    }
    const double *f = G.fx + (i64)g.ix * G.ny + g.jx;
    double f00 = __ldg(f), f01 = __ldg(f + 1), f10 = __ldg(f + G.ny), f11 = __ldg(f + G.ny + 1);
    double low = f00 + g.wx * (f01 - f00), high = f10 + g.wx * (f11 - f10);
    const double ex = low + g.ux * (high - low);
    g.dex_du = high - low;
    g.dex_dw = (1.0 - g.ux) * (f01 - f00) + g.ux * (f11 - f10);
    f = G.fy + (i64)g.iy * (G.ny + 1) + g.jy;
    f00 = __ldg(f);
    f01 = __ldg(f + 1);
    f10 = __ldg(f + G.ny + 1);
    f11 = __ldg(f + G.ny + 2);
    low = f00 + g.wy * (f01 - f00);
    high = f10 + g.wy * (f11 - f10);
    g.ey = low + g.uy * (high - low);
    g.dey_du = high - low;
    g.dey_dw = (1.0 - g.uy) * (f01 - f00) + g.uy * (f11 - f10);
    a[0] = qm * ex;
    if (CYL == 1) {
        a[1] = qm * (g.ey * g.cy);
        a[2] = qm * (g.ey * g.cz);
    } else {
        a[1] = qm * g.ey;
        a[2] = qm * 0.0;
    }
}

// One RK4 step of trace.cu (uniform mesh, gamma = 1), keeping what its reverse needs.
struct StepTape {
    double y[3], w[3];     // the end state
    double a[4][3];        // the stage accelerations
    double u[3][3];        // the stage velocities of stages 2-4
    Stage s[4];            // the stages' field evaluations
    double dt;
    double rate;           // the step size's sensitivity: dt_bar rate (v or a1) joins v's or a1's
    int branch;            // the step size from 0: h, 1: h / |v|, 2: sqrt(2 h / |a|)
};

// Num<true> takes the step size the speed sets and checks that the acceleration's is not
// shorter (trace.cu's `advance`); true where the straight-line step holds.
template <int CYL, bool FAST>
__device__ __forceinline__ bool step_forward(const Grid &G, double qm, double f, const double *x,
                                             const double *v, StepTape &T) {
    Num<FAST> num;
    accel<CYL>(num, G, qm, x, T.a[0], T.s[0]);
    const double *a1 = T.a[0];
    const double v2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    const double a2 = a1[0] * a1[0] + a1[1] * a1[1] + a1[2] * a1[2];
    double y;
    const double speed = num.root(v2, y);
    double dt = num.over_sound(G.h, speed, num.inverse(speed, y));
    int branch = 1;
    if (FAST) {
        num.flag |= !((a2 * G.h) * G.h < (4.0 - 4e-9) * (v2 * v2)) || !(dt > 0.0);
    } else {
        const double accn = sqrt(a2);
        if (!(speed > 0.0)) {
            dt = -1.0;
            branch = 0;
        }
        if (accn > 0.0) {
            const double d2 = sqrt(2.0 * G.h / accn);
            if (dt < 0.0 || d2 < dt) {
                dt = d2;
                branch = 2;
            }
        }
        if (dt < 0.0) {
            dt = G.h;
            branch = 0;
        }
    }
    dt = f * dt;
    T.dt = dt;
    T.branch = branch;
    // (of the step size alone: rounding apart, y^2 is 1 / v^2)
    T.rate = FAST ? -dt * (y * y) : branch == 1 ? -dt / v2 : branch == 2 ? -0.5 * dt / a2 : 0.0;
    const double hdt = 0.5 * dt;
    const double dt6 = num.known(dt, 6.0, 1.0 / 6.0);
    double sx[3], sv[3], kx[3], q[3];  // q: the stage point
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        sx[c] = v[c];
        sv[c] = a1[c];
        q[c] = x[c] + hdt * v[c];
        kx[c] = v[c] + hdt * a1[c];
        T.u[0][c] = kx[c];
    }
    accel<CYL>(num, G, qm, q, T.a[1], T.s[1]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        sx[c] = sx[c] + 2.0 * kx[c];
        sv[c] = sv[c] + 2.0 * T.a[1][c];
        q[c] = x[c] + hdt * kx[c];
        kx[c] = v[c] + hdt * T.a[1][c];
        T.u[1][c] = kx[c];
    }
    accel<CYL>(num, G, qm, q, T.a[2], T.s[2]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        sx[c] = sx[c] + 2.0 * kx[c];
        sv[c] = sv[c] + 2.0 * T.a[2][c];
        q[c] = x[c] + dt * kx[c];
        kx[c] = v[c] + dt * T.a[2][c];
        T.u[2][c] = kx[c];
    }
    accel<CYL>(num, G, qm, q, T.a[3], T.s[3]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        sx[c] = sx[c] + kx[c];
        sv[c] = sv[c] + T.a[3][c];
        T.y[c] = x[c] + dt6 * sx[c];
        T.w[c] = v[c] + dt6 * sv[c];
    }
    // (an intermediate value out of range leaves the end state out of range)
#pragma unroll
    for (int c = 0; c < 3; ++c) num.not_huge(T.y[c]);
    num.not_huge(T.w[0] * T.w[0] + T.w[1] * T.w[1] + T.w[2] * T.w[2]);
    return !num.odd();
}

template <int CYL>
__device__ __noinline__ void step_plain(const Grid &G, double qm, double f, const double *x,
                                        const double *v, StepTape &T) {
    step_forward<CYL, false>(G, qm, f, x, v, T);
}

// The straight-line step, or the IEEE one where it may not hold.
template <int CYL>
__device__ __forceinline__ void step(const Grid &G, double qm, double f, const double *x,
                                     const double *v, StepTape &T) {
    if (!step_forward<CYL, true>(G, qm, f, x, v, T) || G.rh == 0.0) {
        // copies, so that only this branch keeps anything in memory
        const Grid g = G;
        const double x0[3] = {x[0], x[1], x[2]}, v0[3] = {v[0], v[1], v[2]};
        StepTape plain;
        step_plain<CYL>(g, qm, f, x0, v0, plain);
        T = plain;
    }
}

// The edge fields' adjoint, added run by run: consecutive lookups in one cell add into
// registers, a change of cell adds the run to the four edges.
struct Scatter {
    double *fxb, *fyb;
    int ny;
    i64 kx = -1, ky = -1;
    double ax[4] = {0, 0, 0, 0}, ay[4] = {0, 0, 0, 0};

    __device__ __forceinline__ void flush() {
        if (kx >= 0) {
            atomicAdd(fxb + kx, ax[0]);
            atomicAdd(fxb + kx + 1, ax[1]);
            atomicAdd(fxb + kx + ny, ax[2]);
            atomicAdd(fxb + kx + ny + 1, ax[3]);
        }
        if (ky >= 0) {
            atomicAdd(fyb + ky, ay[0]);
            atomicAdd(fyb + ky + 1, ay[1]);
            atomicAdd(fyb + ky + ny + 1, ay[2]);
            atomicAdd(fyb + ky + ny + 2, ay[3]);
        }
        kx = ky = -1;
    }

    __device__ __forceinline__ void add(const Stage &g, double exb, double eyb) {
        const i64 key_x = (i64)g.ix * ny + g.jx;
        if (key_x != kx) {
            if (kx >= 0) {
                atomicAdd(fxb + kx, ax[0]);
                atomicAdd(fxb + kx + 1, ax[1]);
                atomicAdd(fxb + kx + ny, ax[2]);
                atomicAdd(fxb + kx + ny + 1, ax[3]);
            }
            kx = key_x;
            ax[0] = ax[1] = ax[2] = ax[3] = 0.0;
        }
        ax[0] += exb * ((1.0 - g.ux) * (1.0 - g.wx));
        ax[1] += exb * ((1.0 - g.ux) * g.wx);
        ax[2] += exb * (g.ux * (1.0 - g.wx));
        ax[3] += exb * (g.ux * g.wx);
        const i64 key_y = (i64)g.iy * (ny + 1) + g.jy;
        if (key_y != ky) {
            if (ky >= 0) {
                atomicAdd(fyb + ky, ay[0]);
                atomicAdd(fyb + ky + 1, ay[1]);
                atomicAdd(fyb + ky + ny + 1, ay[2]);
                atomicAdd(fyb + ky + ny + 2, ay[3]);
            }
            ky = key_y;
            ay[0] = ay[1] = ay[2] = ay[3] = 0.0;
        }
        ay[0] += eyb * ((1.0 - g.uy) * (1.0 - g.wy));
        ay[1] += eyb * ((1.0 - g.uy) * g.wy);
        ay[2] += eyb * (g.uy * (1.0 - g.wy));
        ay[3] += eyb * (g.uy * g.wy);
    }
};

// The reverse of accel: ab the adjoint of q/m E at q; adds the point's adjoint to qb, and
// exb, eyb get the field's.  Everything but the adjoint is the stage's: no lookup, root or
// quotient stands in the chain of a step's four.
template <int CYL>
__device__ __forceinline__ void accel_reverse(const Grid &G, double qm, const Stage &g,
                                              const double *ab, double *qb,
                                              double &exb, double &eyb) {
    const double ih = G.ih;
    exb = qm * ab[0];
    eyb = CYL == 1 ? qm * fma(ab[1], g.cy, ab[2] * g.cz) : qm * ab[1];
    const double sxb = fma(exb, g.dex_du, eyb * g.dey_du);  // along x (u of either lookup)
    const double syb = fma(exb, g.dex_dw, eyb * g.dey_dw);  // along y / r
    qb[0] = fma(sxb, ih, qb[0]);
    if (CYL == 1) {
        // the unit vector (cy, cz) = (q1, q2) / r
        const double k = qm * g.ey * g.ir;
        const double cyb = k * ab[1], czb = k * ab[2];
        const double rb = syb * ih - fma(cyb, g.cy, czb * g.cz);
        const bool off_axis = g.ir > 0.0;
        qb[1] += off_axis ? fma(rb, g.cy, cyb) : 0.0;
        qb[2] += off_axis ? fma(rb, g.cz, czb) : 0.0;
    } else {
        qb[1] = fma(syb, ih, qb[1]);
    }
}

struct Adj {
    bt_adjoint_args a;
    Grid G;
};

// The checkpoints: every trajectory replayed for its forward steps, its state kept at steps
// 0, kSegment, 2 kSegment, ...; its end state (6, n) for the caller's check.
template <int CYL>
__global__ void __launch_bounds__(kAdjThreads) adjoint_checkpoints(Adj A, double *__restrict__ end) {
    const i64 k = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const bt_adjoint_args &a = A.a;
    if (k >= a.n) return;
    const i64 n = a.n;
    double x[3] = {a.x0[k], a.x0[n + k], a.x0[2 * n + k]};
    double v[3] = {a.v0[k], a.v0[n + k], a.v0[2 * n + k]};
    const i64 steps = a.steps[k];
    const double qm = a.qm[k];
    StepTape T;
    for (i64 s = 0; s < steps; ++s) {
        if (s % kSegment == 0) {
            double *c = a.checkpoints + (s / kSegment) * 6 * n + k;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                c[q * n] = x[q];
                c[(3 + q) * n] = v[q];
            }
        }
        step<CYL>(A.G, qm, a.step_fraction, x, v, T);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            x[q] = T.y[q];
            v[q] = T.w[q];
        }
    }
    if (end) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            end[q * n + k] = x[q];
            end[(3 + q) * n + k] = v[q];
        }
    }
}

// A deposit's place: its radius and the reciprocal, the cell the forward found, the weights
// in it and the radial weight's derivative.
struct Midpoint {
    int i, j;
    double r, ir, u, w, dw_dr;
};

template <int CYL, class N>
__device__ __forceinline__ Midpoint midpoint(N &num, const Grid &G, const double *m) {
    Midpoint M;
    M.r = m[1];
    M.ir = 0.0;
    if (CYL == 1) {
        double y;
        M.r = num.root(m[1] * m[1] + m[2] * m[2], y);
        M.ir = N::fast ? y : 1.0 / M.r;  // used off the axis only
    }
    num.not_tiny(m[0]);
    if (CYL != 1) num.not_tiny(M.r);
    M.i = __double2int_rd(num.known_sound(m[0] - G.ox, G.h, G.rh));
    M.j = __double2int_rd(num.known_sound(M.r - G.oy, G.h, G.rh));
    M.u = num.known_sound(m[0] - (G.ox + G.h * (double)M.i), G.h, G.rh);
    const double low = G.oy + G.h * (double)M.j;
    if (CYL == 1) {
        const double high = low + G.h;
        const double rs = num.div_sound(1.0, high * high - low * low);
        M.w = (M.r * M.r - low * low) * rs;
        M.dw_dr = 2.0 * M.r * rs;
    } else {
        M.w = num.known_sound(M.r - low, G.h, G.rh);
        M.dw_dr = G.ih;
    }
    return M;
}

// The reverse of one step from (x, v): xb, vb hold the adjoint of its end state on entry
// and of its start state on return.  charge_seed: the node charges' adjoint; the hits'
// adjoints of this step's crossings come through hit_seed at the counters cnt.
template <int CYL>
__device__ void step_reverse(const Adj &A, i64 k, double qm, double dq, const double *x,
                             const double *v, double *xb, double *vb,
                             const double *__restrict__ charge_seed,
                             const double *__restrict__ hit_seed, int *cnt, Scatter &sc) {
    const bt_adjoint_args &a = A.a;
    const Grid &G = A.G;
    StepTape T;
    step<CYL>(G, qm, a.step_fraction, x, v, T);
    const double dt = T.dt, hdt = 0.5 * T.dt;
    double yb[3] = {xb[0], xb[1], xb[2]}, wb[3] = {vb[0], vb[1], vb[2]};
    double xs[3] = {0, 0, 0}, vs[3] = {0, 0, 0};  // the start state's adjoint so far
    double dtb = 0.0;

    // the deposit at the step's Hermite midpoint (trace.cu's record, reversed)
    if (charge_seed) {
        double m[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) m[c] = 0.5 * (x[c] + T.y[c]) + dt * (v[c] - T.w[c]) * 0.125;
        Midpoint M;
        {
            Num<true> num;
            M = midpoint<CYL>(num, G, m);
            if (num.odd() || G.rh == 0.0) {
                Num<false> plain;
                M = midpoint<CYL>(plain, G, m);
            }
        }
        int i = M.i, j = M.j;
        double u = M.u, w = M.w, dw_dr = M.dw_dr;
        const double mr = M.r;
        double du_dx = G.ih;
        if (i < 0) {
            u = 0.0;
            i = 0;
            du_dx = 0.0;
        } else if (i >= G.nx - 1) {
            u = 1.0;
            i = G.nx - 2;
            du_dx = 0.0;
        }
        if (j < 0) {
            w = 0.0;
            j = 0;
            dw_dr = 0.0;
        } else if (j >= G.ny - 1) {
            w = 1.0;
            j = G.ny - 2;
            dw_dr = 0.0;
        }
        const i64 node = (i64)i * G.ny + j;
        const double s00 = charge_seed[node], s01 = charge_seed[node + 1];
        const double s10 = charge_seed[node + G.ny], s11 = charge_seed[node + G.ny + 1];
        const double z = s00 * (1.0 - u) * (1.0 - w) + s01 * (1.0 - u) * w +
                         s10 * u * (1.0 - w) + s11 * u * w;
        const double q = dq * dt;
        dtb += dq * z;
        const double ub = q * ((s10 - s00) * (1.0 - w) + (s11 - s01) * w);
        const double wbar = q * ((s01 - s00) * (1.0 - u) + (s11 - s10) * u);
        double mb[3] = {ub * du_dx, 0.0, 0.0};
        const double mrb = wbar * dw_dr;
        if (CYL == 1) {
            if (mr > 0.0) {
                mb[1] = mrb * (m[1] * M.ir);
                mb[2] = mrb * (m[2] * M.ir);
            }
        } else {
            mb[1] = mrb;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            xs[c] += 0.5 * mb[c];
            yb[c] += 0.5 * mb[c];
            vs[c] += dt * 0.125 * mb[c];
            wb[c] -= dt * 0.125 * mb[c];
            dtb += (v[c] - T.w[c]) * 0.125 * mb[c];
        }
    }

    // the plane crossings of the step (the interpolation between its ends, reversed)
    if (hit_seed) {
        for (int p = 0; p < (int)a.n_planes; ++p) {
            const double xp = a.planes[p];
            const double before = x[0] - xp, after = T.y[0] - xp;
            if ((before < 0.0) == (after < 0.0)) continue;
            const int c = --cnt[p];
            if (c < 0 || c >= a.capacity) continue;
            const double *g = hit_seed + ((k * a.n_planes + p) * a.capacity + c) * 8;
            const double den = before - after;
            const double sc_ = before / den;
            double scb = 0.0;
#pragma unroll
            for (int q = 1; q < 3; ++q) {  // the point's y, z
                scb += g[q] * (T.y[q] - x[q]);
                xs[q] += g[q] * (1.0 - sc_);
                yb[q] += g[q] * sc_;
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) {  // the velocity
                scb += g[3 + q] * (T.w[q] - v[q]);
                vs[q] += g[3 + q] * (1.0 - sc_);
                wb[q] += g[3 + q] * sc_;
            }
            xs[0] += scb * (-after / (den * den));
            yb[0] += scb * (before / (den * den));
        }
    }

    // y = x + dt/6 sx, w = v + dt/6 sv
    double sxb[3], svb[3];
    double dt6b = 0.0;
    {
        // sx and sv from the tape: v + 2 u2 + 2 u3 + u4 and a1 + 2 a2 + 2 a3 + a4
        const double dt6 = div_known(dt, 6.0, 1.0 / 6.0);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double sx = v[c] + 2.0 * T.u[0][c] + 2.0 * T.u[1][c] + T.u[2][c];
            const double sv = T.a[0][c] + 2.0 * T.a[1][c] + 2.0 * T.a[2][c] + T.a[3][c];
            xs[c] += yb[c];
            vs[c] += wb[c];
            sxb[c] = dt6 * yb[c];
            svb[c] = dt6 * wb[c];
            dt6b += yb[c] * sx + wb[c] * sv;
        }
    }
    dtb += dt6b / 6.0;
    double u2b[3], u3b[3], u4b[3], a1b[3], a2b[3], a3b[3], a4b[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        vs[c] += sxb[c];
        u2b[c] = 2.0 * sxb[c];
        u3b[c] = 2.0 * sxb[c];
        u4b[c] = sxb[c];
        a1b[c] = svb[c];
        a2b[c] = 2.0 * svb[c];
        a3b[c] = 2.0 * svb[c];
        a4b[c] = svb[c];
    }
    double hdtb = 0.0;
    double qb[3] = {0, 0, 0};
    double exb[4], eyb[4];
    // a4 = acc(q4), q4 = x + dt u3, u4 = v + dt a3
    accel_reverse<CYL>(G, qm, T.s[3], a4b, qb, exb[3], eyb[3]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        vs[c] += u4b[c];
        dtb += u4b[c] * T.a[2][c];
        a3b[c] += dt * u4b[c];
        xs[c] += qb[c];
        dtb += qb[c] * T.u[1][c];
        u3b[c] += dt * qb[c];
        qb[c] = 0.0;
    }
    // a3 = acc(q3), q3 = x + hdt u2, u3 = v + hdt a2
    accel_reverse<CYL>(G, qm, T.s[2], a3b, qb, exb[2], eyb[2]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        vs[c] += u3b[c];
        hdtb += u3b[c] * T.a[1][c];
        a2b[c] += hdt * u3b[c];
        xs[c] += qb[c];
        hdtb += qb[c] * T.u[0][c];
        u2b[c] += hdt * qb[c];
        qb[c] = 0.0;
    }
    // a2 = acc(q2), q2 = x + hdt v, u2 = v + hdt a1
    accel_reverse<CYL>(G, qm, T.s[1], a2b, qb, exb[1], eyb[1]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        vs[c] += u2b[c];
        hdtb += u2b[c] * T.a[0][c];
        a1b[c] += hdt * u2b[c];
        xs[c] += qb[c];
        hdtb += qb[c] * v[c];
        vs[c] += hdt * qb[c];
        qb[c] = 0.0;
    }
    dtb += 0.5 * hdtb;
    // the step size: f h / |v| or f sqrt(2 h / |a1|)
    if (T.branch == 1) {
#pragma unroll
        for (int c = 0; c < 3; ++c) vs[c] += dtb * T.rate * v[c];
    } else if (T.branch == 2) {
#pragma unroll
        for (int c = 0; c < 3; ++c) a1b[c] += dtb * T.rate * T.a[0][c];
    }
    // a1 = acc(x)
    accel_reverse<CYL>(G, qm, T.s[0], a1b, xs, exb[0], eyb[0]);
#pragma unroll
    for (int k4 = 3; k4 >= 0; --k4) sc.add(T.s[k4], exb[k4], eyb[k4]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        xb[c] = xs[c];
        vb[c] = vs[c];
    }
}

// The sweep: every trajectory's steps reversed, from its last to its first.  Bound by the
// latency of one warp a scheduler (250 warps of a design's 8,000 rings): a step's forward
// evaluations keep what their reverse needs, so that the reverse itself is products and sums,
// and run straight-line as the trace's.  8,000 rings of 790 steps at 401 x 101: 3.4 ms with
// the replay (9.7 with a second lookup, IEEE roots and quotients in the reverse, up to 17 for
// a beam whose lengths differ); the checkpoints 1.1 ms (2.1).
template <int CYL>
__global__ void __launch_bounds__(kAdjThreads) adjoint_sweep(Adj A, const double *__restrict__ charge_seed,
                                                             const double *__restrict__ hit_seed,
                                                             double *__restrict__ fx_bar,
                                                             double *__restrict__ fy_bar) {
    const i64 k = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const bt_adjoint_args &a = A.a;
    const i64 n = a.n;
    const bool mine = k < n;
    const i64 steps = mine ? max(a.steps[k], (i64)0) : 0;  // (a count below zero is none)
    int cnt[kMaxPlanes];
    for (int p = 0; p < (int)a.n_planes; ++p) cnt[p] = mine ? (int)a.counts[k * a.n_planes + p] : 0;
    const double qm = mine ? a.qm[k] : 0.0, dq = mine ? a.dq[k] : 0.0;
    Scatter sc{fx_bar, fy_bar, A.G.ny};
    double xb[3] = {0, 0, 0}, vb[3] = {0, 0, 0};
    double tape[kSegment][6];  // the segment's start states
    // The warp walks its longest trajectory's segments together, step by step: lanes whose
    // trajectories have ended wait.  Trip counts of their own let a lane with one segment
    // more replay while its neighbours reversed, each part of the loop run for each: twice
    // the instructions for beams whose step counts straddle a multiple of 64.
    const int segments = (int)((steps + kSegment - 1) / kSegment);
    for (int seg = (int)__reduce_max_sync(0xffffffffu, (unsigned)segments) - 1; seg >= 0; --seg) {
        const int len = (int)max((i64)0, min((i64)kSegment, steps - (i64)seg * kSegment));
        const int longest = (int)__reduce_max_sync(0xffffffffu, (unsigned)len);
        double x[3], v[3];
        if (len > 0) {
            const double *c = a.checkpoints + (i64)seg * 6 * n + k;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                x[q] = c[q * n];
                v[q] = c[(3 + q) * n];
            }
        }
        for (int s = 0; s < longest; ++s) {
            if (s < len) {
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    tape[s][q] = x[q];
                    tape[s][3 + q] = v[q];
                }
                if (s + 1 < len) {
                    StepTape T;
                    step<CYL>(A.G, qm, a.step_fraction, x, v, T);
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        x[q] = T.y[q];
                        v[q] = T.w[q];
                    }
                }
            }
            __syncwarp();
        }
        for (int s = longest - 1; s >= 0; --s) {
            if (s < len) {
                const double xs[3] = {tape[s][0], tape[s][1], tape[s][2]};
                const double vs[3] = {tape[s][3], tape[s][4], tape[s][5]};
                step_reverse<CYL>(A, k, qm, dq, xs, vs, xb, vb, charge_seed, hit_seed, cnt, sc);
            }
            __syncwarp();
        }
    }
    sc.flush();
}

Adj adj_of(const bt_adjoint_args *a) {
    Adj A{};
    A.a = *a;
    A.G = Grid{a->fx, a->fy, (int)a->nx, (int)a->ny, a->origin_x, a->origin_y, a->h,
               sound_origin(a->origin_x) && sound_origin(a->origin_y) ? known_reciprocal(a->h) : 0.0,
               1.0 / a->h};
    return A;
}

void check_args(const bt_adjoint_args *a) {
    BT_REQUIRE(a, "adjoint: null arguments");
    BT_REQUIRE(a->n >= 0, "adjoint: negative trajectory count");
    BT_REQUIRE(a->nx >= 3 && a->ny >= 3, "adjoint: the mesh needs at least 3 nodes per axis");
    BT_REQUIRE(a->nx < (1LL << 30) && a->ny < (1LL << 30), "adjoint: mesh too large");
    BT_REQUIRE(a->cylindrical == 0 || a->cylindrical == 1,
               "adjoint: planar or cylindrical geometry only (no symmetry plane)");
    BT_REQUIRE(a->h > 0.0, "adjoint: h must be positive");
    BT_REQUIRE(a->n_planes >= 0 && a->n_planes <= kMaxPlanes, "adjoint: at most 8 planes");
    BT_REQUIRE(a->segments >= 0, "adjoint: negative checkpoint count");
    if (a->n > 0)
        BT_REQUIRE(a->x0 && a->v0 && a->qm && a->dq && a->steps && a->fx && a->fy &&
                       a->checkpoints && (a->n_planes == 0 || (a->planes && a->counts)),
                   "adjoint: null array");
}

}  // namespace
}  // namespace bt

extern "C" int bt_adjoint_checkpoints(bt_ctx *ctx, const bt_adjoint_args *a, double *end_state) {
    using namespace bt;
    return guarded([&] {
        BT_REQUIRE(ctx, "adjoint: null context");
        check_args(a);
        if (a->n == 0) return;
        const Adj A = adj_of(a);
        Timed timed(ctx, "adjoint_checkpoints");
        const unsigned grid = blocks_for(a->n, kAdjThreads);
        if (a->cylindrical)
            BT_LAUNCH(ctx, adjoint_checkpoints<1>, grid, kAdjThreads, 0, ctx->stream, A, end_state);
        else
            BT_LAUNCH(ctx, adjoint_checkpoints<0>, grid, kAdjThreads, 0, ctx->stream, A, end_state);
        BT_CHECK_LAUNCH();
    });
}

extern "C" int bt_adjoint_sweep(bt_ctx *ctx, const bt_adjoint_args *a, const double *charge_seed,
                                const double *hit_seed, double *fx_bar, double *fy_bar) {
    using namespace bt;
    return guarded([&] {
        BT_REQUIRE(ctx && fx_bar && fy_bar, "adjoint: null argument");
        check_args(a);
        if (a->n == 0 || (!charge_seed && !hit_seed)) return;
        const Adj A = adj_of(a);
        Timed timed(ctx, "adjoint_sweep");
        const unsigned grid = blocks_for(a->n, kAdjThreads);
        if (a->cylindrical)
            BT_LAUNCH(ctx, adjoint_sweep<1>, grid, kAdjThreads, 0, ctx->stream, A, charge_seed,
                      hit_seed, fx_bar, fy_bar);
        else
            BT_LAUNCH(ctx, adjoint_sweep<0>, grid, kAdjThreads, 0, ctx->stream, A, charge_seed,
                      hit_seed, fx_bar, fy_bar);
        BT_CHECK_LAUNCH();
    });
}
