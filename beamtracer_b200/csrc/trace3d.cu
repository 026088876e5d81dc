// The 3D trajectory tracer: kernels/trace_trajectories_3d/trace_trajectories_3d_pyccel.py:19-657
// re-designed for the B200.
//
// One thread per active trajectory advances it by at most `window` steps a launch through
// the staggered edge fields of the patches (finest first, the base mesh last), with a
// magnetic field on the base mesh's nodes, symmetry planes at the lower y and z faces, the
// plane crossings, kept paths, exit and electrode sub-cell tests: the reference's step term
// by term in FP64 with no contracted multiply-add, so a trajectory ends bit for bit where the
// reference's kernel ends it.  Instead of adding to the charge with atomics, the steps write
// their cells' corner shares as records to slots fixed by (window step, trajectory); after
// each window the records are sorted by cell (stable), summed per cell in record order and
// gathered by the nodes, so the node charges are the same on every run.  The current elements
// (has_j) take the same way, one record of three components' eight shares a step (a record a
// share, 24 keys to sort a step, took 119 ms a trace of 100,000 trajectories; 11 ms so).
#include <algorithm>
#include <vector>

#include "common.cuh"

namespace bt {
namespace {

struct Fields3 {
    double e[3], b[3];
};

__device__ __forceinline__ int clamp3(int i, int lo, int hi) { return min(max(i, lo), hi); }

// The first (finest) patch whose node box holds the point, else the base (the last).
__device__ __forceinline__ int finest3(const bt_trace3d_args &a, double p0, double p1, double p2) {
    for (int q = 0; q < (int)a.n_patches - 1; ++q) {
        const double *r = a.patch_real + q * 10;
        if (p0 >= __ldg(r + 4) && p0 <= __ldg(r + 7) && p1 >= __ldg(r + 5) && p1 <= __ldg(r + 8) &&
            p2 >= __ldg(r + 6) && p2 <= __ldg(r + 9))
            return q;
    }
    return (int)a.n_patches - 1;
}

// The reference's nested trilinear form at corner index ci (:231-236).
__device__ __forceinline__ double trilinear(const double *__restrict__ f, i64 ci, int dj, i64 di,
                                            double a, double b, double c) {
    f += ci;
    return (1.0 - a) * ((1.0 - b) * ((1.0 - c) * __ldg(f) + c * __ldg(f + 1)) +
                        b * ((1.0 - c) * __ldg(f + dj) + c * __ldg(f + dj + 1))) +
           a * ((1.0 - b) * ((1.0 - c) * __ldg(f + di) + c * __ldg(f + di + 1)) +
                b * ((1.0 - c) * __ldg(f + di + dj) + c * __ldg(f + di + dj + 1)));
}

// A field box's shape and its edge arrays' offsets.
struct Box3 {
    int nx, ny, nz;
    i64 ofx, ofy, ofz;
};

// E at the point (sx, sy, sz) in cells of a box; s1, s2 the signs a mirror gives.
__device__ __forceinline__ void edges3(const bt_trace3d_args &a, const Box3 &g, double sx, double sy,
                                       double sz, double s1, double s2, double *e) {
    const int pnx = g.nx, pny = g.ny, pnz = g.nz;
    // E_x on (pnx + 1, pny, pnz) at (sx + 1/2, sy, sz)
    double s = sx + 0.5;
    int i = clamp3(__double2int_rd(s), 0, pnx - 1);
    int j = clamp3(__double2int_rd(sy), 0, pny - 2);
    int k = clamp3(__double2int_rd(sz), 0, pnz - 2);
    const int jb = j;
    const double c = sz - (double)k, b = sy - (double)j;
    e[0] = trilinear(a.fxs, g.ofx + ((i64)i * pny + j) * pnz + k, pnz, (i64)pny * pnz, s - (double)i,
                     b, c);
    // E_y on (pnx, pny + 1, pnz) at (sx, sy + 1/2, sz)
    i = clamp3(__double2int_rd(sx), 0, pnx - 2);
    s = sy + 0.5;
    j = clamp3(__double2int_rd(s), 0, pny - 1);
    const double ax = sx - (double)i;
    e[1] = s1 * trilinear(a.fys, g.ofy + ((i64)i * (pny + 1) + j) * pnz + k, pnz,
                          (i64)(pny + 1) * pnz, ax,
                          s - (double)j, c);
    // E_z on (pnx, pny, pnz + 1) at (sx, sy, sz + 1/2)
    s = sz + 0.5;
    k = clamp3(__double2int_rd(s), 0, pnz - 1);
    e[2] = s2 * trilinear(a.fzs, g.ofz + ((i64)i * pny + jb) * (pnz + 1) + k, pnz + 1,
                          (i64)pny * (pnz + 1), ax, b, s - (double)k);
}

// What a trajectory's steps share: the base mesh, its patch, the spacings' reciprocals.
struct Geo3 {
    int nx, ny, nz;   // the base mesh's nodes
    Box3 base;        // the base patch
    i64 first;        // its first charge node
    double h, rh, qm, dq;
};

// A point on the mesh: mirrored below a symmetry plane (with the signs that gives E), in
// cells of the base mesh from its origin.
struct Place3 {
    double p[3], s[3], s1, s2;
};

template <class N>
__device__ __forceinline__ void locate3(N &num, const bt_trace3d_args &a, const Geo3 &G,
                                        const double *q, Place3 &W) {
    W.s1 = W.s2 = 1.0;
    W.p[0] = q[0];
    W.p[1] = q[1];
    W.p[2] = q[2];
    const bool my = a.mirror_y != 0 && q[1] < a.origin_y, mz = a.mirror_z != 0 && q[2] < a.origin_z;
    W.p[1] = my ? 2.0 * a.origin_y - q[1] : q[1];
    W.p[2] = mz ? 2.0 * a.origin_z - q[2] : q[2];
    W.s1 = my ? -1.0 : 1.0;
    W.s2 = mz ? -1.0 : 1.0;
    W.s[0] = num.known(W.p[0] - a.origin_x, G.h, G.rh);
    W.s[1] = num.known(W.p[1] - a.origin_y, G.h, G.rh);
    W.s[2] = num.known(W.p[2] - a.origin_z, G.h, G.rh);
}

// E (from the finest patch holding the point) and B at a place (:173-335).
template <bool HASB, class N>
__device__ __forceinline__ Fields3 fields3(N &num, const bt_trace3d_args &a, const Geo3 &G,
                                           const Place3 &W) {
    Fields3 F;
    if (N::fast) {
        edges3(a, G.base, W.s[0], W.s[1], W.s[2], W.s1, W.s2, F.e);
    } else {
        const int pp = finest3(a, W.p[0], W.p[1], W.p[2]);
        const i64 *pi = a.patch_int + pp * 8;
        const double *pr = a.patch_real + pp * 10;
        const double phh = __ldg(pr + 3);
        const Box3 g{(int)__ldg(pi), (int)__ldg(pi + 1), (int)__ldg(pi + 2),
                     __ldg(pi + 3), __ldg(pi + 4), __ldg(pi + 5)};
        edges3(a, g, (W.p[0] - __ldg(pr)) / phh, (W.p[1] - __ldg(pr + 1)) / phh,
               (W.p[2] - __ldg(pr + 2)) / phh, W.s1, W.s2, F.e);
    }
    F.b[0] = F.b[1] = F.b[2] = 0.0;
    if (HASB) {
        // B on the base mesh's nodes (3, nx, ny, nz), the weights summed in corner order
        const int bi = clamp3(__double2int_rd(W.s[0]), 0, G.nx - 2);
        const int bj = clamp3(__double2int_rd(W.s[1]), 0, G.ny - 2);
        const int bk = clamp3(__double2int_rd(W.s[2]), 0, G.nz - 2);
        const double u = W.s[0] - (double)bi, w = W.s[1] - (double)bj, z = W.s[2] - (double)bk;
        const double wt[8] = {(1.0 - u) * (1.0 - w) * (1.0 - z), (1.0 - u) * (1.0 - w) * z,
                              (1.0 - u) * w * (1.0 - z),         (1.0 - u) * w * z,
                              u * (1.0 - w) * (1.0 - z),         u * (1.0 - w) * z,
                              u * w * (1.0 - z),                 u * w * z};
        const i64 nb = (i64)G.nx * G.ny * G.nz;
        const i64 dj = G.nz, dI = (i64)G.ny * G.nz;
        const i64 base = ((i64)bi * G.ny + bj) * G.nz + bk;
        const i64 off[8] = {0, 1, dj, dj + 1, dI, dI + 1, dI + dj, dI + dj + 1};
        double comp[3];
#pragma unroll
        for (int n0 = 0; n0 < 3; ++n0) {
            const double *bn = a.bn + n0 * nb + base;
            double f = wt[0] * __ldg(bn + off[0]);
#pragma unroll
            for (int q = 1; q < 8; ++q) f = f + wt[q] * __ldg(bn + off[q]);
            comp[n0] = f;
        }
        F.b[0] = W.s1 * W.s2 * comp[0];
        F.b[1] = W.s2 * comp[1];
        F.b[2] = W.s1 * comp[2];
    }
    return F;
}

// 1 / gamma of a proper velocity: 1 with Num<true>, whose steps are not relativistic.
template <class N>
__device__ __forceinline__ double inv_gamma3(N &, double u0, double u1, double u2, double inv_c2) {
    return N::fast ? 1.0 : 1.0 / sqrt(1.0 + (u0 * u0 + u1 * u1 + u2 * u2) * inv_c2);
}

// The relativistic Boris push (J. P. Boris, 1970) of u by the scaled fields e (the kicks)
// and b (the rotation by t = b / gamma, s = 2 t / (1 + t^2)): what the reference's kernel
// calls mpiparticles' relativistic_boris_update for.
template <class N>
__device__ __forceinline__ void boris_push(N &num, double *u, const double *e, const double *b,
                                           double inv_c2) {
    const double m0 = u[0] + e[0], m1 = u[1] + e[1], m2 = u[2] + e[2];
    const double g = N::fast ? 1.0 : sqrt(1.0 + (m0 * m0 + m1 * m1 + m2 * m2) * inv_c2);
    const double t0 = N::fast ? b[0] : b[0] / g, t1 = N::fast ? b[1] : b[1] / g,
                 t2 = N::fast ? b[2] : b[2] / g;
    const double f = num.div_sound(2.0, 1.0 + (t0 * t0 + t1 * t1 + t2 * t2));
    const double s0 = f * t0, s1 = f * t1, s2 = f * t2;
    const double p0 = m0 + (m1 * t2 - m2 * t1);
    const double p1 = m1 + (m2 * t0 - m0 * t2);
    const double p2 = m2 + (m0 * t1 - m1 * t0);
    u[0] = m0 + (p1 * s2 - p2 * s1) + e[0];
    u[1] = m1 + (p2 * s0 - p0 * s2) + e[1];
    u[2] = m2 + (p0 * s1 - p1 * s0) + e[2];
}

// A deposit point's corner node (among `nodes` of a box of (bnx, bny, bnz) from `first`) and
// its trilinear weights, the indices clamped as the reference's (:485-510).
struct Box {
    i64 cc, dj, di;
    double a, b, c;
};

__device__ __forceinline__ void clamp_axis(double s, int n, int &i, double &w) {
    i = __double2int_rd(s);
    w = s - (double)i;
    if (i < 0) {
        w = 0.0;
        i = 0;
    } else if (i >= n - 1) {
        w = 1.0;
        i = n - 2;
    }
}

__device__ __forceinline__ Box box3(i64 first, int bnx, int bny, int bnz, double sx, double sy,
                                    double sz) {
    int i, j, k;
    double a, b, c;
    clamp_axis(sx, bnx, i, a);
    clamp_axis(sy, bny, j, b);
    clamp_axis(sz, bnz, k, c);
    return {first + (i64)i * bny * bnz + (i64)j * bnz + k, bnz, (i64)bny * bnz, a, b, c};
}

// A cell's record: the shares of its eight corners, in the corner order (k, then j, then i
// offsets: q = 4 di + 2 dj + dk) -- of the charge (two 32-byte sectors), or of the current
// element's three components one after the other (six).
template <int N>
struct __align__(64) Rec {
    double c[N];
};
using CellRec = Rec<8>;
using CurrentRec = Rec<24>;

// The eight shares of q, in the reference's corner order (:512-519).
__device__ __forceinline__ void shares8(const Box &B, double q, double *w) {
    const double a = B.a, b = B.b, c = B.c;
    w[0] = (1.0 - a) * (1.0 - b) * (1.0 - c) * q;
    w[1] = (1.0 - a) * (1.0 - b) * c * q;
    w[2] = (1.0 - a) * b * (1.0 - c) * q;
    w[3] = (1.0 - a) * b * c * q;
    w[4] = a * (1.0 - b) * (1.0 - c) * q;
    w[5] = a * (1.0 - b) * c * q;
    w[6] = a * b * (1.0 - c) * q;
    w[7] = a * b * c * q;
}

}  // namespace
}  // namespace bt

namespace bt {
namespace {

struct Trace3 {
    bt_trace3d_args a;
    i64 nx, ny, nz;       // the base mesh's nodes
    int S;                // steps a window
    uint32_t sentinel;    // a slot with no charge record
    uint32_t jsentinel;   // a slot with no current record
};

// The state of a trajectory between steps, as the 2D trace's: its place and the pace it sets
// (the local spacing, the speed's square, the spacing over the speed or -1 at rest), with
// Boris the fields at the last step's end.
struct State3 {
    double x[3], v[3];
    Place3 at;
    double gv, hloc, speed2, dt0;
    Fields3 end;
    bool have;
};

// A step's deposit: its time, its midpoint's box on the charge's patch and on the base mesh.
struct Deposit3 {
    double dt;
    Box charge, mesh;
};

template <class N>
__device__ __forceinline__ void set_pace3(N &num, const bt_trace3d_args &a, const Geo3 &G,
                                          State3 &S) {
    S.gv = inv_gamma3(num, S.v[0], S.v[1], S.v[2], a.inv_c2);
    S.hloc = G.h;
    if (!N::fast) {
        // the spacing of the finest patch at the step's start (:148-163)
        const int q = finest3(a, S.at.p[0], S.at.p[1], S.at.p[2]);
        if (q < (int)a.n_patches - 1) S.hloc = __ldg(a.patch_real + q * 10 + 3);
    }
    double y;
    const double root = num.root(S.v[0] * S.v[0] + S.v[1] * S.v[1] + S.v[2] * S.v[2], y);
    const double speed = N::fast ? root : S.gv * root;
    S.speed2 = speed * speed;
    const double time = num.over_sound(S.hloc, speed, num.inverse(speed, y));
    S.dt0 = speed > 0.0 ? time : -1.0;
}

// q/m (E + v x B) at the velocity u.
template <bool HASB, class N>
__device__ __forceinline__ void pull3(N &, double qm, const Fields3 &F, const double *u, double gk,
                                      double *g) {
    if (N::fast && !HASB) {
        g[0] = qm * F.e[0];
        g[1] = qm * F.e[1];
        g[2] = qm * F.e[2];
    } else if (N::fast) {
        g[0] = qm * (F.e[0] + u[1] * F.b[2] - u[2] * F.b[1]);
        g[1] = qm * (F.e[1] + u[2] * F.b[0] - u[0] * F.b[2]);
        g[2] = qm * (F.e[2] + u[0] * F.b[1] - u[1] * F.b[0]);
    } else {
        g[0] = qm * (F.e[0] + gk * u[1] * F.b[2] - gk * u[2] * F.b[1]);
        g[1] = qm * (F.e[1] + gk * u[2] * F.b[0] - gk * u[0] * F.b[2]);
        g[2] = qm * (F.e[2] + gk * u[0] * F.b[1] - gk * u[1] * F.b[0]);
    }
}

// One step from S to T and its deposit: the 2D trace's `advance` in three dimensions (the
// same straight-line roots and quotients, false where they may not hold, the same step time
// known in advance, `limited` where the acceleration may set it).  With IEEE operations a
// step was 2,429 instructions, its quotients by the spacing and its roots behind one another:
// 509 us a window of 32 Runge-Kutta steps of 100,000 trajectories; 1,620 instructions and 346
// us now, the L1 data path busy 64 % of them with the 96 corner loads a step.  Three blocks a
// multiprocessor (168 registers) hide more of the loads than two with 255 (384 us).  (300,000
// ions turned back at points of their own in 41^3 nodes, whose steps the acceleration limits
// there: 8.7 ms a trace by kTimed, 10.6 by kIeee, 8.8 with IEEE operations throughout.)
enum StepForm3 { kIeee = 0, kSpeculated = 1, kTimed = 2 };

template <int INTEG, bool HASB, StepForm3 FORM>
__device__ __forceinline__ bool advance3(const bt_trace3d_args &a, const Geo3 &G, const State3 &S,
                                         State3 &T, Deposit3 &D, bool &limited) {
    constexpr bool FAST = FORM != kIeee;
    Num<FAST> num;
    const double qm = G.qm, inv_c2 = a.inv_c2, gv = FAST ? 1.0 : S.gv;
    Fields3 F;
    if (INTEG != 0 && S.have)
        F = S.end;
    else
        F = fields3<HASB>(num, a, G, S.at);
    double a1[3];
    pull3<HASB>(num, qm, F, S.v, gv, a1);
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
    dt = a.step_fraction * dt;
    const double hdt = 0.5 * dt;
    double *y = T.x, *w = T.v;
    if (INTEG != 0) {
        // Boris: a half step's kick--rotate--kick, the drift, the second at the end
        const double tau = 0.5 * hdt * qm;
        double u[3] = {S.v[0], S.v[1], S.v[2]};
        double e[3] = {tau * F.e[0], tau * F.e[1], tau * F.e[2]};
        double b[3] = {tau * F.b[0], tau * F.b[1], tau * F.b[2]};
        boris_push(num, u, e, b, inv_c2);
        const double gk = inv_gamma3(num, u[0], u[1], u[2], inv_c2);
#pragma unroll
        for (int c = 0; c < 3; ++c) y[c] = S.x[c] + dt * gk * u[c];
        locate3(num, a, G, y, T.at);
        F = fields3<HASB>(num, a, G, T.at);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            e[c] = tau * F.e[c];
            b[c] = tau * F.b[c];
        }
        boris_push(num, u, e, b, inv_c2);
#pragma unroll
        for (int c = 0; c < 3; ++c) w[c] = u[c];
        T.end = F;
        T.have = true;
    } else {
        const double dt6 = num.known(dt, 6.0, 1.0 / 6.0);
        double sx[3], sv[3], q[3], k[3], g[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sx[c] = gv * S.v[c];
            sv[c] = a1[c];
            q[c] = S.x[c] + hdt * gv * S.v[c];
            k[c] = S.v[c] + hdt * a1[c];
        }
#pragma unroll
        for (int stage = 1; stage < 4; ++stage) {
            Place3 W;
            locate3(num, a, G, q, W);
            F = fields3<HASB>(num, a, G, W);
            const double gk = inv_gamma3(num, k[0], k[1], k[2], inv_c2);
            pull3<HASB>(num, qm, F, k, gk, g);
            const double f = stage == 1 ? hdt : dt;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (stage < 3) {
                    sx[c] = sx[c] + 2.0 * gk * k[c];
                    sv[c] = sv[c] + 2.0 * g[c];
                    q[c] = S.x[c] + f * gk * k[c];
                    k[c] = S.v[c] + f * g[c];
                } else {
                    y[c] = S.x[c] + dt6 * (sx[c] + gk * k[c]);
                    w[c] = S.v[c] + dt6 * (sv[c] + g[c]);
                }
            }
        }
        T.have = false;
        locate3(num, a, G, y, T.at);
    }
    set_pace3(num, a, G, T);
    const double gw = FAST ? 1.0 : T.gv;
    // the space charge dq dt at the step's Hermite midpoint (:451-519); a / 8 is a * 0.125
    double m[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
        m[c] = 0.5 * (S.x[c] + y[c]) + dt * (gv * S.v[c] - gw * w[c]) * 0.125;
    Place3 M;
    locate3(num, a, G, m, M);
    D.mesh = box3(0, G.nx, G.ny, G.nz, M.s[0], M.s[1], M.s[2]);
    if (FAST) {
        D.charge = D.mesh;
        D.charge.cc += G.first;
    } else {
        const int pp = finest3(a, M.p[0], M.p[1], M.p[2]);
        const i64 *pi = a.patch_int + pp * 8;
        const double *pr = a.patch_real + pp * 10;
        const double phh = __ldg(pr + 3);
        D.charge = box3(__ldg(pi + 7), (int)__ldg(pi), (int)__ldg(pi + 1), (int)__ldg(pi + 2),
                        (M.p[0] - __ldg(pr)) / phh, (M.p[1] - __ldg(pr + 1)) / phh,
                        (M.p[2] - __ldg(pr + 2)) / phh);
    }
    D.dt = dt;
#pragma unroll
    for (int c = 0; c < 3; ++c) num.not_huge(y[c]);
    return !num.odd();
}

template <int INTEG, bool HASB>
__device__ __noinline__ void advance3_plain(const bt_trace3d_args &a, const Geo3 &G,
                                            const State3 &S, State3 &T, Deposit3 &D) {
    bool limited;
    advance3<INTEG, HASB, kIeee>(a, G, S, T, D, limited);
}
template <int INTEG, bool HASB>
__device__ __noinline__ bool advance3_timed(const bt_trace3d_args &a, const Geo3 &G,
                                            const State3 &S, State3 &T, Deposit3 &D) {
    bool limited;
    return advance3<INTEG, HASB, kTimed>(a, G, S, T, D, limited);
}

// One window of trajectory m (of the active list): at most S steps from its state.  The
// charge of a run of consecutive steps in one cell is summed into one cell record (key: the
// cell's lower corner node), written to the slot (s n_active + m) of the run's last step s;
// with has_j, each step's current shares go to the slot (s n_active + m) of the current's
// records.  The slots with no record hold the sentinels.  alive[m]: the trajectory has not
// ended (cleared here when it does, with its status written); *live counts the ones still
// going after the window.
// TRY: the straight-line step is tried first, on one patch that is the mesh, without
// relativity; the others take the IEEE operations in line.
template <int INTEG, bool HASB, bool TRY>
__global__ void __launch_bounds__(128, 3) trace3d_window(const __grid_constant__ Trace3 T,
                                                      uint8_t *__restrict__ alive,
                                                      uint32_t *__restrict__ keys,
                                                      CellRec *__restrict__ recs,
                                                      uint32_t *__restrict__ jkeys,
                                                      CurrentRec *__restrict__ jrecs,
                                                      unsigned long long *__restrict__ live) {
    const bt_trace3d_args &a = T.a;
    const i64 m = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const i64 na = a.n_active;
    if (m >= na) return;
    const int S = T.S;
    const bool j_on = a.has_j != 0;
    int s = 0;
    if (alive[m]) {
        const i64 k = a.active[m];
        const i64 n = a.n;
        Geo3 G;
        G.nx = (int)T.nx;
        G.ny = (int)T.ny;
        G.nz = (int)T.nz;
        const i64 *pi = a.patch_int + (a.n_patches - 1) * 8;
        G.base = Box3{G.nx, G.ny, G.nz, __ldg(pi + 3), __ldg(pi + 4), __ldg(pi + 5)};
        G.first = __ldg(pi + 7);
        G.h = a.h;
        G.rh = known_reciprocal(a.h);
        G.qm = a.qm[k];
        G.dq = a.dq[k];
        const double dqk = G.dq;
        State3 now;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            now.x[c] = a.x[c * n + k];
            now.v[c] = a.v[c * n + k];
            now.end.e[c] = now.end.b[c] = 0.0;
        }
        now.have = false;
        {
            Num<false> num;
            locate3(num, a, G, now.x, now.at);
            set_pace3(num, a, G, now);
        }
        const i64 slot = a.path_slot[k];
        i64 ns = a.steps[k];
        i64 st = -1;
        // the current run of steps in one cell: its slot, key and summed shares
        i64 run_slot = -1;
        uint32_t run_key = T.sentinel;
        double run[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (; s < S && ns < a.max_steps; ++s) {
            State3 next;
            Deposit3 D;
            bool ok = false, limited = false;
            if (TRY) ok = advance3<INTEG, HASB, kSpeculated>(a, G, now, next, D, limited);
            if (!TRY) advance3<INTEG, HASB, kIeee>(a, G, now, next, D, limited);
            if (TRY && (!ok || limited)) {
                // copies, so that only this branch keeps anything in memory
                const State3 from = now;
                const Geo3 g = G;
                State3 to;
                Deposit3 d;
                if (!ok || !advance3_timed<INTEG, HASB>(a, g, from, to, d))
                    advance3_plain<INTEG, HASB>(a, g, from, to, d);
                next = to;
                D = d;
            }
            {
                double w[8];
                shares8(D.charge, dqk * D.dt, w);
                const uint32_t key = (uint32_t)D.charge.cc;
                const i64 at = (i64)s * na + m;
                if (run_slot >= 0 && key == run_key) {
                    keys[run_slot] = T.sentinel;  // the run moves on to this step's slot
#pragma unroll
                    for (int q = 0; q < 8; ++q) run[q] = run[q] + w[q];
                } else {
                    if (run_slot >= 0) {
                        keys[run_slot] = run_key;
                        CellRec r;
#pragma unroll
                        for (int q = 0; q < 8; ++q) r.c[q] = run[q];
                        recs[run_slot] = r;
                    }
                    run_key = key;
#pragma unroll
                    for (int q = 0; q < 8; ++q) run[q] = w[q];
                }
                run_slot = at;
                keys[at] = T.sentinel;
            }
            if (j_on) {
                // the current element dq (x' - x) on the base mesh (:520-565)
                double jd[3] = {dqk * (next.x[0] - now.x[0]), dqk * (next.x[1] - now.x[1]),
                                dqk * (next.x[2] - now.x[2])};
                if (a.mirror_y != 0 && 0.5 * (now.x[1] + next.x[1]) < a.origin_y) jd[1] = -jd[1];
                if (a.mirror_z != 0 && 0.5 * (now.x[2] + next.x[2]) < a.origin_z) jd[2] = -jd[2];
                const i64 at = (i64)s * na + m;
                jkeys[at] = (uint32_t)D.mesh.cc;
#pragma unroll
                for (int jc = 0; jc < 3; ++jc) {
                    double w[8];
                    shares8(D.mesh, jd[jc], w);
#pragma unroll
                    for (int q = 0; q < 8; ++q) jrecs[at].c[8 * jc + q] = w[q];
                }
            }
            ns = ns + 1;
            for (i64 p = 0; p < a.n_planes; ++p) {
                const double xp = a.planes[p];
                const double before = now.x[0] - xp, after = next.x[0] - xp;
                if ((before < 0.0) != (after < 0.0)) {
                    const double sc = before / (before - after);
                    i64 *cnt = a.counts + k * a.n_planes + p;
                    const i64 c = *cnt;
                    if (c < a.capacity) {
                        double *hit = a.hits + ((k * a.n_planes + p) * a.capacity + c) * 8;
                        const double gv = now.gv, gw = next.gv;
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
            now = next;
            // the end of the step: off the mesh or in an electrode (:587-641)
            const double px = now.at.p[0], py = now.at.p[1], pz = now.at.p[2];
            if (slot >= 0) {
                const i64 c = a.path_count[slot];
                if (c < a.path_capacity) {
                    double *path = a.paths + (slot * a.path_capacity + c) * 3;
                    path[0] = px;
                    path[1] = py;
                    path[2] = pz;
                }
                a.path_count[slot] = c + 1;
            }
            if (px >= a.upper_x) {
                st = 0;
            } else if (px < a.origin_x) {
                st = 1;
            } else if (py > a.upper_y || py < a.origin_y || pz > a.upper_z || pz < a.origin_z) {
                st = 2;
            } else {
                const double ux = now.at.s[0], uy = now.at.s[1], uz = now.at.s[2];
                const int i = min(__double2int_rz(ux), G.nx - 2);
                const int j = min(__double2int_rz(uy), G.ny - 2);
                const int kz = min(__double2int_rz(uz), G.nz - 2);
                const i64 cell = __ldg(a.cells + ((i64)i * (G.ny - 1) + j) * (G.nz - 1) + kz);
                if (cell >= 0) {
                    const int R = (int)a.refine;
                    const int si = clamp3(__double2int_rz((ux - (double)i) * (double)R), 0, R - 1);
                    const int sj = clamp3(__double2int_rz((uy - (double)j) * (double)R), 0, R - 1);
                    const int sk = clamp3(__double2int_rz((uz - (double)kz) * (double)R), 0, R - 1);
                    const i64 e = __ldg(a.subcells + ((cell * R + si) * R + sj) * R + sk);
                    if (e >= 0) {
                        st = 3;
                        a.electrode[k] = e;
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
            CellRec r;
#pragma unroll
            for (int q = 0; q < 8; ++q) r.c[q] = run[q];
            recs[run_slot] = r;
        }
        if (st == -1 && ns >= a.max_steps) st = 4;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            a.x[c * n + k] = now.x[c];
            a.v[c * n + k] = now.v[c];
        }
        a.steps[k] = ns;
        if (st != -1) {
            a.status[k] = st;
            alive[m] = 0;
        } else {
            atomicAdd(live, 1ull);
        }
    }
    // the slots of the steps not taken hold no record
    for (; s < S; ++s) {
        keys[(i64)s * na + m] = T.sentinel;
        if (j_on) jkeys[(i64)s * na + m] = T.jsentinel;
    }
}

// The cells' sums: the records of a cell lie together after the sort, in runs of hundreds
// where a beam of many trajectories moves down the mesh.  A warp adds 32 records by a
// segmented scan in record order and leaves a cell's sum in the place of one of its records
// (which no other thread reads), that place plus one in `place` (0: a cell of no record): of
// its last record in the cell that is wholly inside the warp, of the warp's last where a cell
// begins here and goes on (`owns` set).  The leading piece of one that began in an earlier
// warp goes to `first` (`ends` set where its cell ends in this warp); cell_chains adds those
// up in warp order.  The sums depend on the records alone.  (One thread a run, waiting for
// each record behind the one before, took 343 us for 1.6 M records in cells of some 500; the
// two kernels take 50 us.)  A window clears a word a cell, which every node reads, and no
// more: with the sums themselves in an array of a record a cell (192 bytes of the current's)
// a window of a hundred trajectories with the current on 257^3 nodes took 2.6 ms and 3.3 GB
// more; 0.6 ms so.
template <int N>
__global__ void __launch_bounds__(256) cell_warps(const uint32_t *__restrict__ K,
                                                  const uint32_t *__restrict__ I, Rec<N> *recs,
                                                  const i64 *__restrict__ count,
                                                  uint32_t *__restrict__ place,
                                                  Rec<N> *__restrict__ first,
                                                  uint8_t *__restrict__ ends,
                                                  uint8_t *__restrict__ owns) {
    const i64 n = *count;
    const i64 w = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w * 32 >= n) return;  // whole warps
    const int lane = threadIdx.x & 31;
    const i64 r = w * 32 + lane;
    const bool valid = r < n;
    const uint32_t key = valid ? K[r] : 0xffffffffu, at = valid ? I[r] : 0u;
    Rec<N> sum;
    if (valid) {
        sum = recs[at];
    } else {
#pragma unroll
        for (int c = 0; c < N; ++c) sum.c[c] = 0.0;
    }
    bool head = valid && (r == 0 || K[r - 1] != key);
    const bool tail = valid && (r + 1 >= n || K[r + 1] != key);
    for (int off = 1; off < 32; off <<= 1) {
        const bool before = __shfl_up_sync(0xffffffffu, head, off);
        const bool add = lane >= off && !head;
#pragma unroll
        for (int c = 0; c < N; ++c) {
            const double v = __shfl_up_sync(0xffffffffu, sum.c[c], off);
            if (add) sum.c[c] = v + sum.c[c];
        }
        if (lane >= off) head = head || before;
    }
    // head: the cell's first record is in this warp
    const bool open = valid && lane == 31 && !tail;
    if (lane == 31) owns[w] = open && head ? 1 : 0;
    if (!tail && !open) return;
    if (head) {
        recs[at] = sum;
        place[key] = at + 1u;
    } else {
        first[w] = sum;
        ends[w] = tail ? 1 : 0;
    }
}

template <int N>
__global__ void __launch_bounds__(256) cell_chains(const uint32_t *__restrict__ I,
                                                   Rec<N> *__restrict__ recs,
                                                   const i64 *__restrict__ count,
                                                   const Rec<N> *__restrict__ first,
                                                   const uint8_t *__restrict__ ends,
                                                   const uint8_t *__restrict__ owns) {
    const i64 n_warps = (*count + 31) / 32;
    // N threads a warp's piece: one a value
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const i64 w0 = t / N;
    const int c = (int)(t - w0 * N);
    if (w0 >= n_warps || !owns[w0]) return;
    double &sum = recs[I[w0 * 32 + 31]].c[c];
    double s = sum;
    for (i64 w = w0 + 1; w < n_warps; ++w) {
        s = s + first[w].c[c];
        if (ends[w]) break;
    }
    sum = s;
}

// A node's shares of the eight cells it is a corner of, added up in a fixed order (the
// corner q = 4 di + 2 dj + dk of the cell at node - (di, dj, dk)), within a box of
// (pnx, pny, pnz) nodes, the node's place in it `local`; a record's components in s.
template <int N>
__device__ __forceinline__ bool corner_sums(const uint32_t *__restrict__ place,
                                            const Rec<N> *__restrict__ recs, i64 node, i64 local,
                                            i64 pnx, i64 pny, i64 pnz, double (&s)[N / 8]) {
    const i64 i = local / (pny * pnz), j = (local / pnz) % pny, k = local % pnz;
    uint32_t at[8], any = 0u;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int di = q >> 2, dj = (q >> 1) & 1, dk = q & 1;
        const i64 ci = i - di, cj = j - dj, ck = k - dk;
        const bool in =
            ci >= 0 && cj >= 0 && ck >= 0 && ci <= pnx - 2 && cj <= pny - 2 && ck <= pnz - 2;
        at[q] = in ? place[node - di * pny * pnz - dj * pnz - dk] : 0u;
        any |= at[q];
    }
#pragma unroll
    for (int m = 0; m < N / 8; ++m) s[m] = 0.0;
    if (any == 0u) return false;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        if (at[q] == 0u) continue;
#pragma unroll
        for (int m = 0; m < N / 8; ++m) s[m] = s[m] + recs[at[q] - 1u].c[8 * m + q];
    }
    return true;
}

__global__ void node_gather3(const uint32_t *__restrict__ place, const CellRec *__restrict__ recs,
                             const i64 *__restrict__ patch_int, int n_patches, i64 n_nodes,
                             double *__restrict__ charge) {
    const i64 node = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= n_nodes) return;
    int p = 0;
    while (p < n_patches - 1 &&
           !(node >= patch_int[p * 8 + 7] && node < patch_int[p * 8 + 7] + patch_int[p * 8 + 6]))
        ++p;
    const i64 *pi = patch_int + p * 8;
    const i64 pnx = pi[0], pny = pi[1], pnz = pi[2], local = node - pi[7];
    if (local < 0 || local >= pnx * pny * pnz) return;
    double s[1];
    if (corner_sums(place, recs, node, local, pnx, pny, pnz, s)) charge[node] += s[0];
}

// The current's three components on the base mesh's nodes.
__global__ void node_gather_current(const uint32_t *__restrict__ place,
                                    const CurrentRec *__restrict__ recs, i64 nx, i64 ny, i64 nz,
                                    double *__restrict__ current) {
    const i64 node = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const i64 n = nx * ny * nz;
    if (node >= n) return;
    double s[3];
    if (!corner_sums(place, recs, node, node, nx, ny, nz, s)) return;
#pragma unroll
    for (int m = 0; m < 3; ++m) current[m * n + node] += s[m];
}

__global__ void fill_flags(uint8_t *__restrict__ flags, i64 n, uint8_t value) {
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) flags[t] = value;
}

}  // namespace
}  // namespace bt

namespace bt {
namespace {

int key_bits(uint64_t max_key) {
    int b = 0;
    while (b < 32 && (max_key >> b) != 0) ++b;
    return b;
}

// A window's records (`slots` keys, those with the sentinel left out) sorted by cell and
// summed per cell in record order, the sums in the records' own places; the returned map of
// n_cells says where (cell_warps).
template <int N>
const uint32_t *sum_cells(bt_ctx *ctx, const uint32_t *keys, Rec<N> *recs, i64 slots,
                          uint32_t sentinel, i64 n_cells) {
    cudaStream_t st = ctx->stream;
    const i64 pieces = (slots + 31) / 32;
    Rec<N> *first = ctx->t3_pieces.as<Rec<N>>(pieces);
    uint8_t *flags = ctx->t3_flags.as<uint8_t>(2 * pieces);
    uint32_t *place = ctx->t3_place.as<uint32_t>(n_cells);
    uint32_t *sk = nullptr, *sv = nullptr;
    const i64 *count = nullptr;
    radix_sort_pairs(ctx, keys, slots, nullptr, key_bits(sentinel), sentinel, &sk, &sv, &count);
    BT_CUDA(cudaMemsetAsync(place, 0, sizeof(uint32_t) * n_cells, st));
    BT_LAUNCH(ctx, cell_warps<N>, blocks_for(pieces * 32, 256), 256, 0, st, sk, sv, recs, count,
              place, first, flags, flags + pieces);
    BT_LAUNCH(ctx, cell_chains<N>, blocks_for(pieces * N, 256), 256, 0, st, sv, recs, count, first,
              flags, flags + pieces);
    BT_CHECK_LAUNCH();
    return place;
}

void trace3d_all(bt_ctx *ctx, const bt_trace3d_args *args, int64_t window) {
    BT_REQUIRE(ctx && args, "trace3d: null argument");
    const bt_trace3d_args &a = *args;
    BT_REQUIRE(a.n_patches >= 1 && a.patch_int && a.patch_real, "trace3d: no patches");
    BT_REQUIRE(a.n_active >= 0 && a.n >= 0, "trace3d: negative sizes");
    BT_REQUIRE(a.capacity >= 0 && a.path_capacity >= 0 && a.n_planes >= 0,
               "trace3d: negative buffer sizes");
    BT_REQUIRE(a.refine >= 1, "trace3d: refine must be positive");
    BT_REQUIRE(a.h > 0.0, "trace3d: h must be positive");
    BT_REQUIRE(a.integrator == 0 || a.integrator == 1, "trace3d: integrator must be 0 or 1");
    BT_REQUIRE(!a.has_b || a.bn, "trace3d: has_b needs bn");
    BT_REQUIRE(!a.has_j || a.current, "trace3d: has_j needs current");
    BT_REQUIRE(a.charge, "trace3d: null charge");
    BT_REQUIRE(a.n_nodes >= 8 && a.n_nodes < (int64_t)0xffffffffLL,
               "trace3d: the charge rows need 8 to 2^32 - 2 nodes");
    if (a.n_active == 0) return;
    Trace3 T;
    T.a = a;
    // the patches' shapes: every deposit key must fall inside the charge rows
    std::vector<int64_t> rows((size_t)8 * a.n_patches);
    BT_CUDA(cudaMemcpyAsync(rows.data(), a.patch_int, sizeof(int64_t) * rows.size(),
                            cudaMemcpyDeviceToHost, ctx->stream));
    BT_CUDA(cudaStreamSynchronize(ctx->stream));
    for (int64_t p = 0; p < a.n_patches; ++p) {
        const int64_t *r = rows.data() + 8 * p;
        BT_REQUIRE(r[0] >= 2 && r[1] >= 2 && r[2] >= 2, "trace3d: a patch needs 2 x 2 x 2 nodes");
        BT_REQUIRE(r[3] >= 0 && r[4] >= 0 && r[5] >= 0 && r[7] >= 0 &&
                       r[7] + r[0] * r[1] * r[2] <= a.n_nodes,
                   "trace3d: a patch's nodes must lie inside the charge rows");
    }
    const int64_t *base = rows.data() + 8 * (a.n_patches - 1);
    T.nx = base[0];
    T.ny = base[1];
    T.nz = base[2];
    BT_REQUIRE(T.nx >= 2 && T.ny >= 2 && T.nz >= 2, "trace3d: the mesh needs 2 x 2 x 2 nodes");
    const i64 nb = T.nx * T.ny * T.nz;
    // one patch that is the mesh, whose spacing has a reciprocal, and no relativity
    bool fast = a.n_patches == 1 && a.inv_c2 == 0.0 && known_reciprocal(a.h) != 0.0;
    if (fast) {
        double row[10];
        BT_CUDA(cudaMemcpyAsync(row, a.patch_real, sizeof(row), cudaMemcpyDeviceToHost, ctx->stream));
        BT_CUDA(cudaStreamSynchronize(ctx->stream));
        fast = row[0] == a.origin_x && row[1] == a.origin_y && row[2] == a.origin_z && row[3] == a.h;
    }
    T.S = window > 0 ? (int)window : 32;
    T.sentinel = (uint32_t)a.n_nodes;
    T.jsentinel = (uint32_t)nb;
    const i64 na = a.n_active;
    const i64 slots = (i64)T.S * na;
    BT_REQUIRE(slots < (i64)0xffffffffLL,
               "trace3d: too many records a window (use a shorter window)");
    uint32_t *keys = ctx->t3_keys.as<uint32_t>(slots);
    CellRec *recs = ctx->t3_vals.as<CellRec>(slots);
    uint32_t *jkeys = a.has_j ? ctx->t3_jkeys.as<uint32_t>(slots) : nullptr;
    CurrentRec *jrecs = a.has_j ? ctx->t3_jvals.as<CurrentRec>(slots) : nullptr;
    uint8_t *alive = ctx->t3_alive.as<uint8_t>(na);
    auto *live = ctx->t3_live.as<unsigned long long>(1);
    unsigned long long *host = static_cast<unsigned long long *>(ctx->host.get(64));
    cudaStream_t st = ctx->stream;
    BT_LAUNCH(ctx, fill_flags, blocks_for(na, 256), 256, 0, st, alive, na, (uint8_t)1);
    // every trajectory ends by max_steps: at most that many windows (and one more)
    const i64 max_windows = a.max_steps / T.S + 2;
    for (i64 w = 0; w < max_windows; ++w) {
        BT_CUDA(cudaMemsetAsync(live, 0, sizeof(unsigned long long), st));
        {
            Timed timed(ctx, "trace3d_window");
#define BT_TRACE3D_CASE(I, B, F)                                                                \
    if ((a.integrator != 0) == (I != 0) && (a.has_b != 0) == B && fast == F)                     \
        BT_LAUNCH(ctx, (trace3d_window<I, B, F>), blocks_for(na, 128), 128, 0, st, T, alive, keys, \
                  recs, jkeys, jrecs, live);
            BT_TRACE3D_CASE(0, false, true) BT_TRACE3D_CASE(0, false, false)
            BT_TRACE3D_CASE(0, true, true) BT_TRACE3D_CASE(0, true, false)
            BT_TRACE3D_CASE(1, false, true) BT_TRACE3D_CASE(1, false, false)
            BT_TRACE3D_CASE(1, true, true) BT_TRACE3D_CASE(1, true, false)
#undef BT_TRACE3D_CASE
        }
        BT_CHECK_LAUNCH();
        // the window's records: sorted by cell, summed per cell, gathered per node
        const uint32_t *place = sum_cells(ctx, keys, recs, slots, T.sentinel, a.n_nodes);
        BT_LAUNCH(ctx, node_gather3, blocks_for(a.n_nodes, 256), 256, 0, st, place, recs,
                  a.patch_int, (int)a.n_patches, a.n_nodes, a.charge);
        if (a.has_j) {
            place = sum_cells(ctx, jkeys, jrecs, slots, T.jsentinel, nb);
            BT_LAUNCH(ctx, node_gather_current, blocks_for(nb, 256), 256, 0, st, place, jrecs, T.nx,
                      T.ny, T.nz, a.current);
        }
        BT_CHECK_LAUNCH();
        BT_CUDA(cudaMemcpyAsync(host, live, sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
        BT_CUDA(cudaStreamSynchronize(st));
        if (*host == 0) return;
    }
    BT_REQUIRE(false, "trace3d: trajectories still live after max_steps steps");
}

}  // namespace
}  // namespace bt

extern "C" int bt_trace_trajectories_3d(bt_ctx *ctx, const bt_trace3d_args *args,
                                        int64_t window) {
    return bt::guarded([&] { bt::trace3d_all(ctx, args, window); });
}
