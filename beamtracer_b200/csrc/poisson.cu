// The field solve on the B200: the finite-volume operator of the reference's field
// (patchwork's NodalPoisson as solver/poisson.py:1-24, 491-534 documents it), solved by
// GMRES preconditioned with a geometric multigrid V-cycle, and Newton's method for the
// Boltzmann plasma species (poisson.py:860-933).
//
// The operator, per free node, A phi = rho / eps0 + c (A = -laplacian, FD-scaled rows):
// Shortley-Weller rows with the bracketed surface distances at nodes with four cells, the
// cut edge's two-point flux at nodes on a face, (1 -/+ 1/2j) radial weights and 4 (phi_1 -
// phi_0) on the axis, mirror images on Neumann faces; fixed nodes keep their values.
//
// Multigrid: vertex-centred coarsening (coarse node I at fine node 2I, the last coarse
// node on the last fine node), bilinear prolongation P that is zero at fixed fine nodes,
// Galerkin coarse operators A_1 = P^T W A_0 P (W the control volumes, which make W A_0
// nearly symmetric) and A_{l+1} = P^T A_l P: 9-point stencils on every coarse level, built
// on the device (and rebuilt for every Newton step's Jacobian).  Smoothing: red-black
// Gauss-Seidel on the 5-point fine level, four-colour Gauss-Seidel on the 9-point levels;
// the coarsest level (at most 256 nodes) is inverted from its band's LU factors, or by a
// pivoting Gauss-Jordan where those meet a tiny pivot.
#include <cmath>
#include <vector>

#include "common.cuh"

namespace bt {
namespace {

constexpr int kCoarsest = 256;  // the coarsest level is inverted densely (at most this size)
constexpr double kEps0 = 8.8541878188e-12;  // scipy.constants.epsilon_0 (CODATA 2022)

struct Axis {
    i64 n = 0, nc = 0;
    bool coarsened = false;
    Buffer lo, w;        // per fine node: coarse index and its weight
    Buffer r0, rw;       // per coarse node: its first fine node and kRestrict weights from there
};

constexpr int kRestrict = 4;  // fine nodes per axis that one coarse node restricts from

struct Level {
    i64 nx = 0, ny = 0, n = 0;
    Buffer c4;      // level 0: cw, ce, cs, cn (4 n)
    Buffer diag;    // level 0: the diagonal (with the reaction)
    Buffer base;    // level 0: the diagonal without the reaction
    Buffer rdiag;   // the reciprocal of the diagonal (a smoothing update multiplies by it)
    Buffer weight;  // level 0: the control volumes W
    Buffer a9;      // coarse levels: 9 coefficients per node, (dI + 1) * 3 + (dJ + 1)
    Buffer active;  // uint8: free (level 0) or a nonzero row (coarse)
    Buffer x, b;
    Buffer x2;              // the second x of staged smoothing (it writes the other buffer)
    double *cur = nullptr;  // which of x, x2 holds the level's x while a V-cycle is recorded
    Axis ax, ay;            // the map to the next coarser level
};

// -- the fine operator (mirrors oracle/poisson.py:coefficients) ---------------------------

__global__ void build_fine(i64 nx, i64 ny, const double *__restrict__ x, double h, int cyl,
                           i64 j0, const uint8_t *__restrict__ fixed, const double *__restrict__ dist,
                           double g0, double g1, double g2, double g3,
                           double *__restrict__ c4, double *__restrict__ base,
                           double *__restrict__ src, double *__restrict__ weight,
                           uint8_t *__restrict__ active) {
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const i64 n = nx * ny;
    if (t >= n) return;
    const i64 i = t / ny, j = t - i * ny;
    const double h_lo = i > 0 ? x[i] - x[i - 1] : 0.0;
    const double h_hi = i < nx - 1 ? x[i + 1] - x[i] : 0.0;
    const double ax = dist[t], bx = dist[n + t], ay = dist[2 * n + t], by = dist[3 * n + t];
    const bool four = i > 0 && i < nx - 1 && j > 0 && j < ny - 1;
    double cw = 0.0, ce = 0.0, cs = 0.0, cn = 0.0, s = 0.0;
    // x
    if (i > 0 && i < nx - 1) {
        const double dm = ax * h_lo, dp = bx * h_hi;
        if (four) {
            cw = 2.0 / ((dm + dp) * dm);
            ce = 2.0 / ((dm + dp) * dp);
        } else {
            const double L = 0.5 * (h_lo + h_hi);
            cw = 1.0 / (L * dm);
            ce = 1.0 / (L * dp);
        }
    } else if (i == 0) {
        ce = 2.0 / (h_hi * (bx * h_hi));
        s += 2.0 * g0 / h_hi;
    } else {
        cw = 2.0 / (h_lo * (ax * h_lo));
        s += 2.0 * g1 / h_lo;
    }
    // y
    const bool mid = j > 0 && j < ny - 1;
    if (!cyl) {
        const double dm = ay * h, dp = by * h;
        if (mid) {
            if (four) {
                cs = 2.0 / ((dm + dp) * dm);
                cn = 2.0 / ((dm + dp) * dp);
            } else {
                cs = 1.0 / (h * dm);
                cn = 1.0 / (h * dp);
            }
        } else if (j == 0) {
            cn = 2.0 / (h * dp);
            s += 2.0 * g2 / h;
        } else {
            cs = 2.0 / (h * dm);
            s += 2.0 * g3 / h;
        }
    } else {
        // the radial index of the row: j0 = r_0 / h for a refined patch off the axis
        const double jj = j + j0 > 1 ? (double)(j + j0) : 1.0;
        const double h2 = h * h;
        if (mid) {
            if (four) {
                cs = (2.0 / ay - 1.0 / jj) / ((ay + by) * h2);
                cn = (2.0 / by + 1.0 / jj) / ((ay + by) * h2);
            } else {
                cs = (1.0 - 0.5 / jj) / (ay * h2);
                cn = (1.0 + 0.5 / jj) / (by * h2);
            }
        } else if (j == 0) {
            // the axis; off the axis (a patch's side inside the domain, a row the
            // composite operator does not use) a face row
            cn = (j0 == 0 ? 4.0 : 2.0) / (by * h2);
        } else {
            cs = 2.0 / (ay * h2);
            s += (1.0 + 0.5 / jj) * 2.0 * g3 / h;
        }
    }
    const bool free = fixed[t] == 0;
    c4[t] = free ? cw : 0.0;
    c4[n + t] = free ? ce : 0.0;
    c4[2 * n + t] = free ? cs : 0.0;
    c4[3 * n + t] = free ? cn : 0.0;
    base[t] = free ? cw + ce + cs + cn : 1.0;
    src[t] = free ? s : 0.0;
    active[t] = free ? 1 : 0;
    // the control volume (divided by 2 pi in cylindrical geometry)
    const double lx = 0.5 * (h_lo + h_hi);  // half an edge at an x face
    double ly = (j > 0 && j < ny - 1) ? h : 0.5 * h;
    if (cyl) ly = j + j0 == 0 ? 0.125 * h * h : (double)(j + j0) * h * ly;
    weight[t] = lx * ly;
}

// The transposed operator, scaled by the control volumes: B = W^-1 A^T W, whose
// neighbour coefficients are B[t][nb] = A[nb][t] W_nb / W_t (A[nb][t] the coefficient of
// the neighbour's row pointing back at t; zero for a held node's row or a held neighbour,
// whose rows hold none); the diagonal stays.  W A is symmetric away from the cut rows next
// to electrodes and the faces, so B equals A there and the multigrid built for A serves
// it: A^T z = g is solved as B y = W^-1 g, z = W y.
__global__ void transpose_c4(i64 nx, i64 ny, const double *__restrict__ c4,
                             const double *__restrict__ weight,
                             const uint8_t *__restrict__ active, double *__restrict__ c4t) {
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const i64 n = nx * ny;
    if (t >= n) return;
    const i64 i = t / ny, j = t - i * ny;
    const bool free = active[t] != 0;
    const double wt = weight[t];
    c4t[t] = free && i > 0 ? c4[n + (t - ny)] * weight[t - ny] / wt : 0.0;  // west's east
    c4t[n + t] = free && i < nx - 1 ? c4[t + ny] * weight[t + ny] / wt : 0.0;  // east's west
    c4t[2 * n + t] = free && j > 0 ? c4[3 * n + (t - 1)] * weight[t - 1] / wt : 0.0;
    c4t[3 * n + t] = free && j < ny - 1 ? c4[2 * n + (t + 1)] * weight[t + 1] / wt : 0.0;
}

// v <- v / W (divide) or v * W on the free nodes: to and from the scaled transposed system.
__global__ void scale_by_weight(i64 n, const double *__restrict__ weight,
                                const uint8_t *__restrict__ active, int divide,
                                double *__restrict__ v) {
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n || !active[t]) return;
    v[t] = divide ? v[t] / weight[t] : v[t] * weight[t];
}

// The sensitivity to the held potentials of a quantity whose sensitivity to phi is
// phi_bar, given z = A_ff^-T phi_bar (free nodes): the free rows read the held neighbours'
// potentials through their coefficients, so out_d = phi_bar_d + sum over the free
// neighbours i of c(i -> d) z_i; 0 on free nodes.
__global__ void fixed_adjoint(i64 nx, i64 ny, const double *__restrict__ c4,
                              const uint8_t *__restrict__ active, const double *__restrict__ z,
                              const double *__restrict__ phi_bar, double *__restrict__ out) {
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const i64 n = nx * ny;
    if (t >= n) return;
    if (active[t]) {
        out[t] = 0.0;
        return;
    }
    const i64 i = t / ny, j = t - i * ny;
    double s = phi_bar[t];
    if (i < nx - 1 && active[t + ny]) s += c4[t + ny] * z[t + ny];              // east's west
    if (i > 0 && active[t - ny]) s += c4[n + (t - ny)] * z[t - ny];             // west's east
    if (j < ny - 1 && active[t + 1]) s += c4[2 * n + (t + 1)] * z[t + 1];       // north's south
    if (j > 0 && active[t - 1]) s += c4[3 * n + (t - 1)] * z[t - 1];            // south's north
    out[t] = s;
}

__global__ void add_diag(i64 n, const double *__restrict__ base, const double *__restrict__ reaction,
                         const uint8_t *__restrict__ active, double *__restrict__ diag,
                         double *__restrict__ rdiag) {
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const double d = base[t] + ((reaction && active[t]) ? reaction[t] : 0.0);
    diag[t] = d;
    rdiag[t] = 1.0 / d;
}

// -- Galerkin coarse operator -----------------------------------------------------------

struct Fine {
    i64 nx, ny;
    const double *c4, *diag, *a9, *weight;  // c4/diag for the 5-point level, a9 otherwise
    const uint8_t *active;
    const int32_t *lox, *loy;
    const double *wx, *wy;
    const int32_t *rx0, *ry0;  // restriction: first fine node of each coarse node
    const double *rxw, *ryw;   //   and kRestrict weights from it (zero: not a neighbour)
    i64 ncx, ncy;
};

// The weights of the coarse nodes I - 1, I, I + 1 at the kRestrict + 2 fine nodes from
// first - 1 on (zero off the axis).
__device__ __forceinline__ void axis_weights(const int32_t *__restrict__ lo,
                                             const double *__restrict__ w, i64 n, int first, int I,
                                             double (&p)[kRestrict + 2][3]) {
#pragma unroll
    for (int a = 0; a < kRestrict + 2; ++a) {
        const int k = first - 1 + a;
        const bool in = k >= 0 && k < (int)n;
        const int l = in ? lo[k] : -4;
        const double v = in ? w[k] : 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d)
            p[a][d] = l == I + d - 1 ? v : (l + 1 == I + d - 1 ? 1.0 - v : 0.0);
    }
}

// A thread a coarse node.  Its row is a product over the axes: with the weights of both
// axes in registers, each fine row's three neighbour rows are contracted along y, then
// along x -- some 54 multiply-adds a fine node and no branch but the fine node's own, and
// the loads of a fine row of nodes are all in flight together.  PLAIN adds every neighbour
// to all nine coarse nodes one after another (see update9).  Testing every pair of fine
// neighbour and coarse node instead (a branch and an index a term) took 60 us a level of a
// 1025 x 513 mesh, its levels of a few thousand nodes as long as the finest; the product
// takes 22 us for the finest and 14 for the others.
constexpr int kGalerkinThreads = 64;

template <bool NINE, bool PLAIN>
__global__ void __launch_bounds__(kGalerkinThreads)
    galerkin(Fine F, double *__restrict__ a9c, double *__restrict__ rdiag_c,
             uint8_t *__restrict__ active_c) {
    const i64 nc = F.ncx * F.ncy, n = F.nx * F.ny;
    const int t = blockIdx.x * kGalerkinThreads + threadIdx.x;
    if (t >= nc) return;
    const int ny = (int)F.ny, ncy = (int)F.ncy;
    const int I = t / ncy, J = t - I * ncy;
    const int k0 = F.rx0[I], l0 = F.ry0[J];
    double px[kRestrict + 2][3], py[kRestrict + 2][3], acc[3][3];
    axis_weights(F.lox, F.wx, F.nx, k0, I, px);
    axis_weights(F.loy, F.wy, F.ny, l0, J, py);
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int e = 0; e < 3; ++e) acc[d][e] = 0.0;
    // 1 where a fine node is in the mesh and free
    auto free_at = [&](int k, int l) {
        return k >= 0 && k < (int)F.nx && l >= 0 && l < ny && F.active[(i64)k * ny + l] ? 1.0 : 0.0;
    };
#pragma unroll
    for (int a = 0; a < kRestrict; ++a) {
        const double pk = px[a + 1][1];
        if (pk == 0.0) continue;
        const int k = k0 + a;
#pragma unroll
        for (int c = 0; c < kRestrict; ++c) {
            const double pl = py[c + 1][1];
            const int l = l0 + c;
            if (pl == 0.0 || free_at(k, l) == 0.0) continue;
            const i64 f = (i64)k * ny + l;
            const double wgt = pk * pl * (F.weight ? F.weight[f] : 1.0);
            double m[3][3];  // the fine row, held neighbours left out
            if (NINE) {
#pragma unroll
                for (int d = 0; d < 3; ++d)
#pragma unroll
                    for (int e = 0; e < 3; ++e)
                        m[d][e] = F.a9[(i64)(3 * d + e) * n + f] * free_at(k + d - 1, l + e - 1);
            } else {
                m[0][0] = m[0][2] = m[2][0] = m[2][2] = 0.0;
                m[1][1] = F.diag[f];
                m[0][1] = -F.c4[f] * free_at(k - 1, l);
                m[2][1] = -F.c4[n + f] * free_at(k + 1, l);
                m[1][0] = -F.c4[2 * n + f] * free_at(k, l - 1);
                m[1][2] = -F.c4[3 * n + f] * free_at(k, l + 1);
            }
            if (PLAIN) {
                // every neighbour (d, e), in row order, to every coarse node (p, q) it
                // prolongs from
#pragma unroll
                for (int d = 0; d < 3; ++d)
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        if (!NINE && d != 1 && e != 1) continue;
                        const double t = wgt * m[d][e];
#pragma unroll
                        for (int p = 0; p < 3; ++p) {
                            const double tp = t * px[a + d][p];
#pragma unroll
                            for (int q = 0; q < 3; ++q) acc[p][q] += tp * py[c + e][q];
                        }
                    }
                continue;
            }
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                double row[3];
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    row[d] = fma(m[d][0], py[c][e], fma(m[d][1], py[c + 1][e], m[d][2] * py[c + 2][e]));
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    acc[d][e] = fma(wgt, fma(px[a][d], row[0],
                                             fma(px[a + 1][d], row[1], px[a + 2][d] * row[2])),
                                    acc[d][e]);
            }
        }
    }
    const bool on = acc[1][1] != 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int e = 0; e < 3; ++e)
            a9c[(i64)(3 * d + e) * nc + t] = on ? acc[d][e] : (d == 1 && e == 1 ? 1.0 : 0.0);
    rdiag_c[t] = on ? 1.0 / acc[1][1] : 1.0;
    active_c[t] = on ? 1 : 0;
}

// -- smoothing, residual, transfer ---------------------------------------------------------

// A Gauss-Seidel update of a node from its neighbours, on a 5-point row (coefficients west,
// east, south, north) or a 9-point row (the eight neighbours' in row order).  Two chains of
// fused multiply-adds and the diagonal's reciprocal: a colour phase is one such update a
// thread between barriers, so its time is the update's latency -- 17 dependent roundings
// and an IEEE quotient, some 240 cycles, before; some 56 so.  Every form of a
// single solve's smoothing (a launch a colour, staged tiles, the coarse levels in one
// launch) takes these updates.
// PLAIN: one term after another and the quotient by the diagonal (rd is the diagonal).  A
// batch of candidates takes PLAIN throughout (smoothing, restriction, the coarse operators
// and their inverse): some of its candidates never settle, and such a one multiplies a
// rounding of its field by 1e5 and more over its iterations -- with the fused forms some
// sweeps end with moments 3.5e-8 from PLAIN's (the others within 2e-12).  The batch's launches
// are many tiles deep, so the longer chains cost it little: 360 ms a sweep for 352.
template <bool PLAIN = false>
__device__ __forceinline__ double update5(double b, double cw, double ce, double cs, double cn,
                                          double xw, double xe, double xs, double xn, double rd) {
    if (PLAIN) return (b + cw * xw + ce * xe + cs * xs + cn * xn) / rd;
    return (fma(ce, xe, fma(cw, xw, b)) + fma(cn, xn, cs * xs)) * rd;
}
template <bool PLAIN = false>
__device__ __forceinline__ double update9(double b, const double (&a)[8], const double (&x)[8],
                                          double rd) {
    if (PLAIN) {
#pragma unroll
        for (int q = 0; q < 8; ++q) b -= a[q] * x[q];
        return b / rd;
    }
    const double p = fma(-a[3], x[3], fma(-a[2], x[2], fma(-a[1], x[1], fma(-a[0], x[0], b))));
    const double q = fma(a[7], x[7], fma(a[6], x[6], fma(a[5], x[5], a[4] * x[4])));
    return (p - q) * rd;
}

__global__ void smooth5(i64 nx, i64 ny, const double *__restrict__ c4,
                        const double *__restrict__ rdiag, const uint8_t *__restrict__ active,
                        const double *__restrict__ b, double *__restrict__ x, int colour) {
    const i64 n = nx * ny;
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    // thread t handles the t-th node of the colour
    const i64 half = (ny + 1) / 2;
    const i64 i = t / half;
    if (i >= nx) return;
    const i64 j = 2 * (t - i * half) + ((i + colour) & 1);
    if (j >= ny) return;
    const i64 f = i * ny + j;
    if (!active[f]) return;
    x[f] = update5(b[f], c4[f], c4[n + f], c4[2 * n + f], c4[3 * n + f], i > 0 ? x[f - ny] : 0.0,
                   i < nx - 1 ? x[f + ny] : 0.0, j > 0 ? x[f - 1] : 0.0,
                   j < ny - 1 ? x[f + 1] : 0.0, rdiag[f]);
}

// The nodes of one of four colours (i % 2, j % 2) of a 9-point level: item t of `count`.
__host__ __device__ __forceinline__ i64 colour_count(i64 nx, i64 ny, int colour) {
    const int ci = colour >> 1, cj = colour & 1;
    return ((nx - ci + 1) / 2) * ((ny - cj + 1) / 2);
}

__global__ void smooth9(i64 nx, i64 ny, const double *__restrict__ a9,
                        const double *__restrict__ rdiag, const uint8_t *__restrict__ active,
                        const double *__restrict__ b, double *__restrict__ x, int colour) {
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= colour_count(nx, ny, colour)) return;
    const i64 n = nx * ny;
    const int ci = colour >> 1, cj = colour & 1;
    const i64 hy = (ny - cj + 1) / 2;
    const i64 i = 2 * (t / hy) + ci, j = 2 * (t % hy) + cj;
    const i64 f = i * ny + j;
    if (!active[f]) return;
    double a[8], v[8];
#pragma unroll
    for (int q = 0, k = 0; q < 9; ++q) {
        if (q == 4) continue;
        const i64 i2 = i + q / 3 - 1, j2 = j + q % 3 - 1;
        a[k] = a9[(i64)q * n + f];
        v[k++] = i2 >= 0 && i2 < nx && j2 >= 0 && j2 < ny ? x[i2 * ny + j2] : 0.0;
    }
    x[f] = update9(b[f], a, v, rdiag[f]);
}

// -- smoothing staged through shared memory -------------------------------------------------
//
// One launch runs up to kMaxPhases colour phases of Gauss-Seidel on a tile of interior
// nodes plus a halo as wide as the phases (phase k is exact on the halo's rings k + 1 and
// inward, so after the last phase the interior is exactly what per-colour launches give).
// The tile's coefficients, right-hand side, active flags and x are read from global memory
// once, each phase then runs from shared memory, and the interior is written to a second x
// buffer: no block reads what another block of the same launch writes.  Coefficients and b
// are stored compacted by colour, so the threads of a phase read consecutive words; x keeps
// the tile's natural layout.
constexpr int kMaxPhases = 8;
constexpr int kStageThreads = 512;
constexpr int kStage5X = 32, kStage5Y = 32;  // 5-point level: interior rows x columns
constexpr int kStage9X = 16, kStage9Y = 32;  // 9-point levels

struct Phases {
    int count;
    int colour[kMaxPhases];
};

// Where a V-cycle reads its right-hand side and leaves its result: held on the device, so
// that one captured graph serves every vector (a Krylov step sets them to its basis vector
// and its image) without a copy in and out of the level's own.
struct CycleIo {
    const double *b;
    double *z;
};

// The halo of `count` phases: rounded up to even, so the tile's origin has even (i, j)
// and a node's colour follows from its place in the tile.
__host__ __device__ inline int stage_halo(int count) { return (count + 1) & ~1; }

// (P xc)[f], the prolongation of the coarse correction xc to the fine node f of an active
// fine node (the bilinear weights of the fine node's coarse neighbours, in (sx, sy) order).
__device__ __forceinline__ double prolong_sum(const Fine &F, i64 f, const double *xc) {
    const i64 k = f / F.ny, l = f - k * F.ny;
    const i64 ix = F.lox[k], iy = F.loy[l];
    const double wx = F.wx[k], wy = F.wy[l];
    double s = 0.0;
    for (int sx = 0; sx < 2; ++sx) {
        const double px = sx ? 1.0 - wx : wx;
        if (px == 0.0 || ix + sx >= F.ncx) continue;
        for (int sy = 0; sy < 2; ++sy) {
            const double py = sy ? 1.0 - wy : wy;
            if (py == 0.0 || iy + sy >= F.ncy) continue;
            s += px * py * xc[(ix + sx) * F.ncy + iy + sy];
        }
    }
    return s;
}

__host__ __device__ inline size_t stage_smem(bool nine, int tx, int ty, int halo) {
    const size_t m = (size_t)(tx + 2 * halo) * (ty + 2 * halo);
    return m * sizeof(double) * (nine ? 11 : 7) + m;
}

// One tile (bx, by) of a batch's staged smoothing, for the tile sizes and phase counts that no
// register tile is compiled for, in PLAIN arithmetic (update9).
template <bool NINE, int R>
__device__ __forceinline__ void smooth_staged_tile(
    i64 nx, i64 ny, const double *__restrict__ c4, const double *__restrict__ diag,
    const double *__restrict__ a9, const uint8_t *__restrict__ active,
    const double *__restrict__ b, const double *__restrict__ xin, double *__restrict__ xout,
    int tx, int ty, const Phases &ph, const Fine &F, const double *__restrict__ xc, i64 bx,
    i64 by, bool zero_in = false) {
    // zero_in: x starts at zero (xin is not read)
    // xc, when not NULL: the coarse correction, prolonged onto x as it is read (the values
    // prolong_add would leave in xin)
    extern __shared__ double sm[];
    constexpr int Q = NINE ? 9 : 5;
    constexpr int K = NINE ? 4 : 2;  // colours
    const int halo = stage_halo(ph.count);
    const int wx = tx + 2 * halo, wy = ty + 2 * halo, m = wx * wy, per = m / K, hy = wy / 2;
    const int tid = threadIdx.x, nt = blockDim.x;
    double *coef = sm;          // [Q][m], position slot(a, c)
    double *bs = coef + Q * m;  // [m], position slot(a, c)
    double *xs = bs + m;        // [m], natural a * wy + c
    uint8_t *act = reinterpret_cast<uint8_t *>(xs + m);
    // the compacted position of tile node (a, c): its colour's block, then its index there
    auto slot = [&](int a, int c) -> int {
        if (NINE) return (((a & 1) << 1) | (c & 1)) * per + (a >> 1) * hy + (c >> 1);
        return ((a + c) & 1) * per + ((a * wy + c) >> 1);
    };
    const i64 i0 = bx * tx - halo, j0 = by * ty - halo;
    const i64 n = nx * ny;
    // Every array of a node is loaded at once, whether or not the node is active (the
    // flag selects afterwards): one round trip to memory a node, not two.  An inactive
    // node's coefficients are stored but never read.
#pragma unroll 4
    for (int e = tid; e < m; e += nt) {
        const int a = e / wy, c = e - a * wy;
        const i64 i = i0 + a, j = j0 + c;
        const int pos = slot(a, c);
        double xv = 0.0, bv = 0.0;
        uint8_t av = 0;
        if (i >= 0 && i < nx && j >= 0 && j < ny) {
            const i64 f = i * ny + j;
            xv = zero_in ? 0.0 : xin[f];
            av = active[f];
            const double bf = b[f];
            if (NINE) {
                double q9[9];
#pragma unroll
                for (int q = 0; q < 9; ++q) q9[q] = a9[(i64)q * n + f];
#pragma unroll
                for (int q = 0; q < 9; ++q) coef[q * m + pos] = q9[q];
            } else {
                double q5[5];
#pragma unroll
                for (int q = 0; q < 4; ++q) q5[q] = c4[(i64)q * n + f];
                q5[4] = diag[f];
#pragma unroll
                for (int q = 0; q < 5; ++q) coef[q * m + pos] = q5[q];
            }
            if (av) {
                if (xc) xv = xv + prolong_sum(F, f, xc);
                bv = bf;
            }
        }
        xs[e] = xv;
        bs[pos] = bv;
        act[pos] = av;
    }
    __syncthreads();
    // The nodes this thread updates: node u = tid + r nt of each colour's compacted list,
    // with its place in x's layout and its ring (its distance from the tile's edge; -1 for
    // a node it never updates: past the list, outside the mesh, or held).  A neighbour
    // outside the mesh holds x = 0 in the tile and adds nothing: no bounds tests.
    int xi[K][R], ring[K][R];
#pragma unroll
    for (int k = 0; k < K; ++k) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int u = tid + r * nt;
            int a = 0, c = 0;
            if (NINE) {
                const int ua = u / hy;
                a = 2 * ua + (k >> 1);
                c = 2 * (u - ua * hy) + (k & 1);
            } else {
                a = u / hy;
                c = 2 * (u - a * hy) + ((a + k) & 1);
            }
            const i64 i = i0 + a, j = j0 + c;
            const bool mine = u < per && i >= 0 && i < nx && j >= 0 && j < ny && act[k * per + u];
            xi[k][r] = a * wy + c;
            ring[k][r] = mine ? min(min(a, wx - 1 - a), min(c, wy - 1 - c)) : -1;
        }
    }
    for (int kk = 0; kk < ph.count; ++kk) {
        const int colour = ph.colour[kk];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (k != colour) continue;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (ring[k][r] <= kk) continue;  // phase kk is exact from ring kk + 1 inward
                const int pos = k * per + tid + r * nt, q = xi[k][r];
                if (NINE) {
                    const double c[8] = {coef[pos],         coef[m + pos],     coef[2 * m + pos],
                                         coef[3 * m + pos], coef[5 * m + pos], coef[6 * m + pos],
                                         coef[7 * m + pos], coef[8 * m + pos]};
                    const double v[8] = {xs[q - wy - 1], xs[q - wy],     xs[q - wy + 1], xs[q - 1],
                                         xs[q + 1],      xs[q + wy - 1], xs[q + wy],     xs[q + wy + 1]};
                    xs[q] = update9<true>(bs[pos], c, v, coef[4 * m + pos]);
                } else {
                    xs[q] = update5<true>(bs[pos], coef[pos], coef[m + pos], coef[2 * m + pos],
                                    coef[3 * m + pos], xs[q - wy], xs[q + wy], xs[q - 1], xs[q + 1],
                                    coef[4 * m + pos]);
                }
            }
        }
        __syncthreads();
    }
    for (int e = tid; e < tx * ty; e += nt) {
        const int ea = e / ty;
        const int a = halo + ea, c = halo + (e - ea * ty);
        const i64 i = i0 + a, j = j0 + c;
        if (i < nx && j < ny) xout[i * ny + j] = xs[a * wy + c];
    }
}

// -- the same smoothing with the coefficients in registers ----------------------------------
//
// A tile whose sizes the compiler knows.  A thread has one node of each colour (R of them),
// whose coefficients, right-hand side and reciprocal diagonal it loads straight into
// registers -- all of its nodes' loads in flight together, no index that is not a shift --
// and only x goes through shared memory: a phase is eight (four) shared loads, the update and
// a store.  Staging the coefficients through shared memory at sizes known at run time spent
// 1,760 instructions a warp, most on indices, for some 300 of arithmetic: 10.3 us a launch of
// a 9-point level, whatever its size, against 5.5 before the coarse correction and 6.3 after
// it, and 12.0 for the finest level of 801 x 201 against 7.9 and 10.0.

// One side of a fine-coarse pair's prolongation, as build_axis lays it out: the lower coarse
// neighbour of fine node k and its weight.
struct CoarseAxis {
    int n, nc;
};
__device__ __forceinline__ int coarse_low(const CoarseAxis &A, int k, double &w) {
    if (A.n <= 3) {
        w = 1.0;
        return k;
    }
    const int I = min(k >> 1, A.nc - 2);
    const int c1 = min(2 * I + 2, A.n - 1);
    w = c1 - 2 * I == 2 ? 0.5 * (double)(c1 - k) : (double)(c1 - k);
    return I;
}

// A level as the smoother reads it.
struct SmoothView {
    int nx, ny;
    i64 n;
    const double *c4, *rdiag, *a9, *b, *xin, *xc;  // xin NULL: from zero; xc NULL: no correction
    const uint8_t *active;
    double *xout;
    CoarseAxis ax, ay;  // to the next level (with xc)
};

template <bool NINE, int TX, int TY, int COUNT>
struct Tile {
    static constexpr int halo = (COUNT + 1) & ~1;
    static constexpr int wx = TX + 2 * halo, wy = TY + 2 * halo;
    static constexpr int colours = NINE ? 4 : 2;
    static constexpr int per = wx * wy / colours;       // nodes of a colour
    static constexpr int r = (per + 511) / 512;         // a thread's nodes of a colour
    static constexpr int threads = ((per + r - 1) / r + 31) / 32 * 32;
};

// PLAIN: rdiag names the diagonal itself (update9).
template <bool NINE, int TX, int TY, int COUNT, bool REVERSE, bool PLAIN = false>
__device__ __forceinline__ void smooth_tile(const SmoothView &L, int bx, int by) {
    using S = Tile<NINE, TX, TY, COUNT>;
    constexpr int K = S::colours, R = S::r, WX = S::wx, WY = S::wy, HY = WY / 2;
    constexpr int Q = NINE ? 8 : 4;
    __shared__ double xs[WX * WY];
    const int tid = threadIdx.x, i0 = bx * TX - S::halo, j0 = by * TY - S::halo;
    double coef[K][R][Q], b[K][R], rd[K][R], x[K][R];
    int at[K][R], ring[K][R];  // the node's place in xs; its distance from the tile's edge, or
                               // -1 where it is never updated (held, or outside the mesh)
#pragma unroll
    for (int k = 0; k < K; ++k) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int u = tid + r * S::threads;
            const int ua = u / HY, uc = u - ua * HY;
            const int a = NINE ? 2 * ua + (k >> 1) : ua;
            const int c = NINE ? 2 * uc + (k & 1) : 2 * uc + ((a + k) & 1);
            const int i = i0 + a, j = j0 + c;
            const bool in = u < S::per && i >= 0 && i < L.nx && j >= 0 && j < L.ny;
            const int f = in ? i * L.ny + j : 0;
            at[k][r] = a * WY + c;
            const uint8_t act = L.active[f];
            ring[k][r] = in && act ? min(min(a, WX - 1 - a), min(c, WY - 1 - c)) : -1;
            if (NINE) {
#pragma unroll
                for (int q = 0; q < 8; ++q) coef[k][r][q] = L.a9[(q < 4 ? q : q + 1) * L.n + f];
            } else {
#pragma unroll
                for (int q = 0; q < Q; ++q) coef[k][r][q] = L.c4[q * L.n + f];
            }
            rd[k][r] = L.rdiag[f];
            b[k][r] = L.b[f];
            x[k][r] = in && L.xin ? L.xin[f] : 0.0;
            if (L.xc && in && act) {
                // the prolonged correction, in the order prolong_sum adds it
                double wx, wy;
                const int I = coarse_low(L.ax, i, wx), J = coarse_low(L.ay, j, wy);
                double sum = 0.0;
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    const double px = d ? 1.0 - wx : wx;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const double py = e ? 1.0 - wy : wy;
                        if (px != 0.0 && py != 0.0) sum += px * py * L.xc[(I + d) * L.ay.nc + J + e];
                    }
                }
                x[k][r] += sum;
            }
            if (u < S::per) xs[at[k][r]] = x[k][r];
        }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < COUNT; ++kk) {
        const int k = REVERSE ? K - 1 - kk % K : kk % K;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (ring[k][r] > kk) {  // phase kk is exact from ring kk + 1 inward
                const double *q = xs + at[k][r];
                const double(&c)[Q] = coef[k][r];
                if constexpr (NINE) {
                    const double v[8] = {q[-WY - 1], q[-WY], q[-WY + 1], q[-1],
                                         q[1],       q[WY - 1], q[WY],   q[WY + 1]};
                    x[k][r] = update9<PLAIN>(b[k][r], c, v, rd[k][r]);
                } else {
                    x[k][r] = update5<PLAIN>(b[k][r], c[0], c[1], c[2], c[3], q[-WY], q[WY], q[-1],
                                             q[1], rd[k][r]);
                }
                xs[at[k][r]] = x[k][r];
            }
        }
        if (kk + 1 < COUNT) __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int a = at[k][r] / WY, c = at[k][r] - a * WY;
            const int i = i0 + a, j = j0 + c;
            if (tid + r * S::threads < S::per && a >= S::halo && a < S::halo + TX && c >= S::halo &&
                c < S::halo + TY && i < L.nx && j < L.ny)
                L.xout[i * L.ny + j] = x[k][r];
        }
    }
}

template <bool NINE, int TX, int TY, int COUNT, bool REVERSE>
__global__ void __launch_bounds__(Tile<NINE, TX, TY, COUNT>::threads)
    smooth_level(SmoothView L, const CycleIo *__restrict__ io, bool first, bool last) {
    // io: the finest level's smoothing, which starts the cycle from its b and ends it in z
    if (io) {
        L.b = io->b;
        if (last) L.xout = io->z;
    }
    if (first) L.xin = nullptr;
    smooth_tile<NINE, TX, TY, COUNT, REVERSE>(L, blockIdx.x, blockIdx.y);
}

// y = A x (level 0, 5-point) on active rows, 0 elsewhere; with b: r = b - A x.  Node f of
// an (nx, ny) level; returns y[f].
__device__ __forceinline__ double apply5_item(i64 f, i64 nx, i64 ny, const double *__restrict__ c4,
                                              const double *__restrict__ diag,
                                              const uint8_t *__restrict__ active,
                                              const double *__restrict__ x,
                                              const double *__restrict__ b,
                                              double *__restrict__ y) {
    const i64 n = nx * ny;
    if (!active[f]) {
        y[f] = 0.0;
        return 0.0;
    }
    const i64 i = f / ny, j = f - i * ny;
    double s = diag[f] * x[f];
    if (i > 0) s -= c4[f] * x[f - ny];
    if (i < nx - 1) s -= c4[n + f] * x[f + ny];
    if (j > 0) s -= c4[2 * n + f] * x[f - 1];
    if (j < ny - 1) s -= c4[3 * n + f] * x[f + 1];
    const double out = b ? b[f] - s : s;
    y[f] = out;
    return out;
}

// -- the residual and its restriction -----------------------------------------------------
//
// One launch a level: a block forms the residual of the fine nodes around kRestrictX x
// kRestrictY coarse nodes, a thread a fine node with its row's loads all in flight, weighs
// it (by the control volumes on level 0) into shared memory, and adds up each coarse node's
// nine from there, the weights from build_axis's rule.  The blocks' edges are computed twice
// (10 % of the rows); the residual never goes to memory and there is one launch of 4.2 us (5.1
// for the finest level) where the two took 8 (the restriction alone 4.8: its nine loads
// waited for table entries).
constexpr int kRestrictX = 8, kRestrictY = 16;
constexpr int kRestrictFineX = 2 * kRestrictX + 1, kRestrictFineY = 2 * kRestrictY + 1;
constexpr int kRestrictThreads = (kRestrictFineX * kRestrictFineY + 31) / 32 * 32;

struct RestrictView {
    int nx, ny, ncx, ncy;
    i64 n;
    const double *c4, *diag, *a9, *weight;  // level 0: c4, diag and weight; else a9
    const uint8_t *active;
    const double *x, *b;
    double *bc;
};

// The weight of coarse node I at fine node k of an axis.
__device__ __forceinline__ double coarse_weight(const CoarseAxis &A, int k, int I) {
    double w;
    const int lo = coarse_low(A, k, w);
    return I == lo ? w : (I == lo + 1 ? 1.0 - w : 0.0);
}

// PLAIN: every sum one term after another, as a batch of candidates restricts.
template <bool NINE, bool PLAIN = false>
__device__ __forceinline__ void restrict_tile(const RestrictView &L, int bx, int by) {
    __shared__ double rs[kRestrictFineX * kRestrictFineY];
    const int tid = threadIdx.x, nx = L.nx, ny = L.ny;
    const int I0 = bx * kRestrictX, J0 = by * kRestrictY;
    const int k0 = nx > 3 ? 2 * I0 - 1 : I0 - 1, l0 = ny > 3 ? 2 * J0 - 1 : J0 - 1;
    if (tid < kRestrictFineX * kRestrictFineY) {
        const int i = k0 + tid / kRestrictFineY, j = l0 + tid % kRestrictFineY;
        double r = 0.0;
        if (i >= 0 && i < nx && j >= 0 && j < ny) {
            const int f = i * ny + j;
            const bool w = i > 0, e = i < nx - 1, s = j > 0, n = j < ny - 1;
            const double *x = L.x + f;
            if (NINE) {
                double a[9];
#pragma unroll
                for (int q = 0; q < 9; ++q) a[q] = L.a9[q * L.n + f];
                const double v[9] = {w && s ? x[-ny - 1] : 0.0, w ? x[-ny] : 0.0,
                                     w && n ? x[-ny + 1] : 0.0, s ? x[-1] : 0.0,
                                     x[0],                      n ? x[1] : 0.0,
                                     e && s ? x[ny - 1] : 0.0,  e ? x[ny] : 0.0,
                                     e && n ? x[ny + 1] : 0.0};
                if (PLAIN) {
                    r = L.b[f];
#pragma unroll
                    for (int k = 0; k < 9; ++k) r -= a[k] * v[k];
                } else {
                    double p = L.b[f], q = a[5] * v[5];
#pragma unroll
                    for (int k = 0; k < 5; ++k) p = fma(-a[k], v[k], p);
#pragma unroll
                    for (int k = 6; k < 9; ++k) q = fma(a[k], v[k], q);
                    r = p - q;
                }
            } else if (PLAIN) {
                double t = L.diag[f] * x[0];
                t -= L.c4[f] * (w ? x[-ny] : 0.0);
                t -= L.c4[L.n + f] * (e ? x[ny] : 0.0);
                t -= L.c4[2 * L.n + f] * (s ? x[-1] : 0.0);
                t -= L.c4[3 * L.n + f] * (n ? x[1] : 0.0);
                r = (L.b[f] - t) * L.weight[f];
            } else {
                const double p = fma(-L.diag[f], x[0], L.b[f]);
                const double q = fma(L.c4[f], w ? x[-ny] : 0.0, L.c4[L.n + f] * (e ? x[ny] : 0.0));
                const double u = fma(L.c4[2 * L.n + f], s ? x[-1] : 0.0,
                                     L.c4[3 * L.n + f] * (n ? x[1] : 0.0));
                r = (p + (q + u)) * L.weight[f];
            }
            if (!L.active[f]) r = 0.0;
        }
        rs[tid] = r;
    }
    __syncthreads();
    if (tid >= kRestrictX * kRestrictY) return;
    const int I = I0 + tid / kRestrictY, J = J0 + tid % kRestrictY;
    if (I >= L.ncx || J >= L.ncy) return;
    const CoarseAxis ax{nx, L.ncx}, ay{ny, L.ncy};
    const int ki = nx > 3 ? 2 * I : I, li = ny > 3 ? 2 * J : J;  // the middle of the nine
    double sum = 0.0;
#pragma unroll
    for (int d = -1; d <= 1; ++d) {
        const double pk = ki + d >= 0 && ki + d < nx ? coarse_weight(ax, ki + d, I) : 0.0;
        double row = 0.0;
#pragma unroll
        for (int e = -1; e <= 1; ++e) {
            const double pl = li + e >= 0 && li + e < ny ? coarse_weight(ay, li + e, J) : 0.0;
            if (pl == 0.0 || pk == 0.0) continue;
            const double r = rs[(ki + d - k0) * kRestrictFineY + (li + e - l0)];
            if (PLAIN)
                sum += pk * pl * r;
            else
                row = fma(pl, r, row);
        }
        if (!PLAIN) sum = fma(pk, row, sum);
    }
    L.bc[I * L.ncy + J] = sum;
}

template <bool NINE>
__global__ void __launch_bounds__(kRestrictThreads)
    restrict_level(RestrictView L, const CycleIo *__restrict__ io) {
    if (io) L.b = io->b;
    restrict_tile<NINE>(L, blockIdx.x, blockIdx.y);
}

__global__ void fill_zero(i64 n, double *__restrict__ x) {
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f < n) x[f] = 0.0;
}

__global__ void prolong_add(Fine F, const double *__restrict__ xc, double *__restrict__ x) {
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= F.nx * F.ny) return;
    if (F.active[f]) x[f] = x[f] + prolong_sum(F, f, xc);
}

// The coarsest level: the dense matrix of its 9-point operator, inverted in place in `M`
// (global memory, n x n) by Gauss-Jordan with partial pivoting, one block.  The pivot is the
// largest |M[r][k]| (the first such row).  `status` is set to 1 on a zero pivot (a singular
// operator: no node of the mesh is held).
constexpr int kInvertThreads = 1024;

// The coarsest operator is a 9-point stencil: ordered along its shorter side first its
// matrix is banded with half-bandwidth b = min(nx, ny) + 1 (at most 17 for 256 nodes), and
// its LU factors without pivoting fit shared memory (n rows of 2b + 1).  One block
// factorises it, a warp a row and a lane a column of the moving b x b window, one barrier a
// step: the multipliers stay unscaled until the end (every thread scales its own by the
// step's reciprocal pivot), so no step waits for a scaled column.  A second kernel then
// solves L U x = e_c with a thread a column, the b unknowns a row still touches in registers
// (right-looking: b independent multiply-adds a row, the factors' columns read from shared
// memory by all lanes at once), into the dense inverse the V-cycle applies.  The work is one
// serial chain of 3 n rows, so the time is rows times latency: with the substitutions
// reading global memory row by row and a serial scan of every pivot row, 208 nodes
// (b = 9, an 801 x 201 mesh) took 374 us and 153 nodes (b = 10, 1025 x 513) 284 us; now
// 49 + 94 us in PLAIN's order, which a linear operator takes, and 28 + 32 us for the 153 of
// a Newton step's.  A pivot smaller than 1e-12 of its row (a matrix that needs pivoting, or a
// singular one) sets *fallback and the pivoting Gauss-Jordan below computes the inverse
// instead.
constexpr int kBandMax = 17;
constexpr int kBandPad = kBandMax + 1;  // a factor column's stride, in doubles (even: 16-byte loads)
constexpr int kSolveThreads = 32;       // columns a block of coarsest_band_solve: a warp

__host__ __device__ __forceinline__ int band_half(i64 nx, i64 ny) {
    return (int)(nx < ny ? nx : ny) + 1;
}

__host__ __device__ __forceinline__ size_t band_smem(i64 nx, i64 ny) {
    return sizeof(double) * (size_t)(nx * ny) * (size_t)(2 * band_half(nx, ny) + 2);
}

// The node at place o of the band's order and the other way round.
__device__ __forceinline__ int band_order(int node, int nx, int ny) {
    return nx < ny ? (node % ny) * nx + node / ny : node;
}
__device__ __forceinline__ int band_node(int o, int nx, int ny) {
    return nx < ny ? (o % nx) * ny + o / nx : o;
}

// factors: column k of L below the diagonal at [k kBandPad + j - 1] (row k + j), column k of
// U above it at [(n + k) kBandPad + j - 1] (row k - j), the reciprocal pivots after both.
// PLAIN (see update9) divides by the pivots, keeps row k of U right of the diagonal (column
// k + j) in the place of its column, and the pivots themselves.
template <bool PLAIN>
__global__ void __launch_bounds__(32 * kBandMax) coarsest_band_factor(
    int nx, int ny, const double *__restrict__ a9, double *__restrict__ factors,
    int *__restrict__ fallback) {
    extern __shared__ double band[];  // row r: band[r * W + (c - r + b)], |c - r| <= b
    const int n = nx * ny;
    const int b = band_half(nx, ny), W = 2 * b + 1;
    double *inv = band + n * W;  // the pivots' reciprocals; PLAIN: the pivots
    const auto over = [](double v, double d) { return PLAIN ? v / d : v * d; };
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    for (int e = tid; e < n * W; e += nt) band[e] = 0.0;
    __syncthreads();
    for (int node = tid; node < n; node += nt) {
        const int i = node / ny, j = node % ny, r = band_order(node, nx, ny);
        for (int di = -1; di <= 1; ++di)
            for (int dj = -1; dj <= 1; ++dj) {
                const int i2 = i + di, j2 = j + dj;
                if (i2 < 0 || i2 >= nx || j2 < 0 || j2 >= ny) continue;
                const int c = band_order(i2 * ny + j2, nx, ny);
                band[r * W + (c - r + b)] = a9[(i64)((di + 1) * 3 + (dj + 1)) * n + node];
            }
    }
    __syncthreads();
    // row k + 1 + warp, column k + 1 + lane of step k's window
    double *mine = band + (warp + 1) * W + b + lane - warp;
    const double *left = band + (warp + 1) * W + b - 1 - warp, *up = band + b + 1 + lane;
    const double *diag = band + b;
    for (int k = 0; k < n; ++k) {
        const double r = PLAIN ? *diag : 1.0 / *diag;
        if (tid == 0) inv[k] = r;
        if (lane < b && k + 1 + lane < n && k + 1 + warp < n)
            *mine = PLAIN ? *mine - (*left / r) * *up : fma(-(*left * r), *up, *mine);
        __syncthreads();
        mine += W;
        left += W;
        up += W;
        diag += W;
    }
    for (int k = tid; k < n; k += nt) {
        const double r = inv[k];
        double row = 0.0;
        double *L = factors + k * kBandPad, *U = factors + (n + k) * kBandPad;
        for (int j = 1; j <= kBandPad; ++j) {
            const bool below = j <= b && k + j < n, above = j <= b && k - j >= 0;
            L[j - 1] = below ? over(band[(k + j) * W + b - j], r) : 0.0;
            U[j - 1] = PLAIN ? (below ? band[k * W + b + j] : 0.0)
                             : (above ? band[(k - j) * W + b + j] : 0.0);
            // row k's own entries: its multipliers and its part of U
            if (above) row = fmax(row, fabs(over(band[k * W + b - j], inv[k - j])));
            if (below) row = fmax(row, fabs(band[k * W + b + j]));
        }
        const double piv = band[k * W + b];
        row = fmax(row, fabs(piv));
        if (!(fabs(piv) > 1e-12 * row)) *fallback = 1;
        factors[2 * n * kBandPad + k] = r;
    }
}

// M[., col] = (L U)^-1 e_col, a thread a column: KB at least b, even.  The window w[j] holds
// row o + j's (forward) or o - j's (backward) remaining right-hand side; PLAIN's backward one
// row o + 1 + j's solution, a row's terms taken from the diagonal outwards.  The forward
// results go through M; the backward pass reads its own column's values kAhead rows early.
template <int KB, bool PLAIN>
__global__ void __launch_bounds__(kSolveThreads) coarsest_band_solve(
    int nx, int ny, const double *__restrict__ factors, double *__restrict__ M,
    const int *__restrict__ fallback) {
    extern __shared__ __align__(16) double f[];
    if (*fallback) return;
    const int n = nx * ny;
    // the first KB of every factor column (PLAIN: of U, row), then the (reciprocal) pivots
    for (int e = threadIdx.x; e < 2 * n * KB; e += kSolveThreads) {
        const int k = e / KB;
        f[e] = factors[k * kBandPad + (e - k * KB)];
    }
    double *inv = f + 2 * n * KB;
    for (int e = threadIdx.x; e < n; e += kSolveThreads) inv[e] = factors[2 * n * kBandPad + e];
    __syncthreads();
    const int col = blockIdx.x * kSolveThreads + threadIdx.x;
    const int oc = col < n ? band_order(col, nx, ny) : -1;
    double w[KB + 1];
#pragma unroll
    for (int j = 0; j <= KB; ++j) w[j] = 0.0;
    for (int o = 0; o < n; ++o) {
        const double y = o == oc ? w[0] + 1.0 : w[0];
        const double2 *L = reinterpret_cast<const double2 *>(f + o * KB);
#pragma unroll
        for (int j = 0; j < KB / 2; ++j) {
            const double2 l = L[j];
            w[2 * j] = PLAIN ? w[2 * j + 1] - l.x * y : fma(-l.x, y, w[2 * j + 1]);
            w[2 * j + 1] = PLAIN ? w[2 * j + 2] - l.y * y : fma(-l.y, y, w[2 * j + 2]);
        }
        w[KB] = 0.0;
        if (col < n) M[(i64)band_node(o, nx, ny) * n + col] = y;
    }
    constexpr int kAhead = 8;
    double ahead[kAhead];
#pragma unroll
    for (int q = 0; q < kAhead; ++q)
        ahead[q] = col < n && n - 1 - q >= 0 ? M[(i64)band_node(n - 1 - q, nx, ny) * n + col] : 0.0;
#pragma unroll
    for (int j = 0; j <= KB; ++j) w[j] = 0.0;
    for (int top = n - 1; top >= 0; top -= kAhead) {
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const int o = top - q;
            if (o < 0) break;
            double x = PLAIN ? ahead[q] : (w[0] + ahead[q]) * inv[o];
            const int next = o - kAhead;
            ahead[q] = col < n && next >= 0 ? M[(i64)band_node(next, nx, ny) * n + col] : 0.0;
            const double2 *U = reinterpret_cast<const double2 *>(f + (n + o) * KB);
#pragma unroll
            for (int j = 0; j < KB / 2; ++j) {
                const double2 u = U[j];
                if (PLAIN) {
                    x -= u.x * w[2 * j];
                    x -= u.y * w[2 * j + 1];
                } else {
                    w[2 * j] = fma(-u.x, x, w[2 * j + 1]);
                    w[2 * j + 1] = fma(-u.y, x, w[2 * j + 2]);
                }
            }
            if (PLAIN) {
                x = x / inv[o];
#pragma unroll
                for (int j = KB; j > 0; --j) w[j] = w[j - 1];
                w[0] = x;
            } else {
                w[KB] = 0.0;
            }
            if (col < n) M[(i64)band_node(o, nx, ny) * n + col] = x;
        }
    }
}

__global__ void __launch_bounds__(kInvertThreads) coarsest_invert(
    i64 nx, i64 ny, const double *__restrict__ a9, double *M, int *__restrict__ status,
    const int *__restrict__ fallback) {
    if (fallback && *fallback == 0) return;  // the banded factorisation made the inverse
    __shared__ int perm[kCoarsest];
    __shared__ double best_v[kInvertThreads / 32];
    __shared__ int best_r[kInvertThreads / 32];
    __shared__ int pivot_row;
    const int n = (int)(nx * ny);
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    for (int e = tid; e < n * n; e += nt) {
        const int row = e / n, col = e % n;
        const i64 i = row / ny, j = row % ny, i2 = col / ny, j2 = col % ny;
        const i64 di = i2 - i, dj = j2 - j;
        double v = 0.0;
        if (di >= -1 && di <= 1 && dj >= -1 && dj <= 1)
            v = a9[(i64)((di + 1) * 3 + (dj + 1)) * n + row];
        M[e] = v;
    }
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        // the pivot: a block-wide arg-max of |M[r][k]|, r >= k, the lowest r on ties
        double v = -1.0;
        int r = n;
        for (int q = k + tid; q < n; q += nt) {
            const double a = fabs(M[(i64)q * n + k]);
            if (a > v) {
                v = a;
                r = q;
            }
        }
        for (int off = 16; off > 0; off >>= 1) {
            const double v2 = __shfl_down_sync(0xffffffffu, v, off);
            const int r2 = __shfl_down_sync(0xffffffffu, r, off);
            if (v2 > v || (v2 == v && r2 < r)) {
                v = v2;
                r = r2;
            }
        }
        if (lane == 0) {
            best_v[warp] = v;
            best_r[warp] = r;
        }
        __syncthreads();
        if (tid == 0) {
            double bv = best_v[0];
            int br = best_r[0];
            for (int w = 1; w < nt / 32; ++w)
                if (best_v[w] > bv || (best_v[w] == bv && best_r[w] < br)) {
                    bv = best_v[w];
                    br = best_r[w];
                }
            if (br >= n) br = k;
            pivot_row = br;
            perm[k] = br;
            if (!(bv > 0.0)) *status = 1;
        }
        __syncthreads();
        const int p = pivot_row;
        if (p != k)
            for (int c = tid; c < n; c += nt) {
                const double t = M[(i64)k * n + c];
                M[(i64)k * n + c] = M[(i64)p * n + c];
                M[(i64)p * n + c] = t;
            }
        __syncthreads();
        const double piv = M[(i64)k * n + k];
        __syncthreads();
        for (int c = tid; c < n; c += nt) M[(i64)k * n + c] = (c == k ? 1.0 : M[(i64)k * n + c]) / piv;
        __syncthreads();
        for (int e = tid; e < n * n; e += nt) {
            const int rr = e / n, c = e % n;
            if (rr == k || c == k) continue;
            M[e] -= M[(i64)rr * n + k] * M[(i64)k * n + c];
        }
        __syncthreads();
        for (int rr = tid; rr < n; rr += nt)
            if (rr != k) M[(i64)rr * n + k] = -M[(i64)rr * n + k] * M[(i64)k * n + k];
        __syncthreads();
    }
    for (int k = n - 1; k >= 0; --k) {
        const int p = perm[k];
        if (p != k)
            for (int rr = tid; rr < n; rr += nt) {
                const double t = M[(i64)rr * n + k];
                M[(i64)rr * n + k] = M[(i64)rr * n + p];
                M[(i64)rr * n + p] = t;
            }
        __syncthreads();
    }
}

// x = inv b on the active rows, 0 on held ones (the inverse's held rows are unit rows up to
// the rounding that pivoting mixes into them; a correction never moves a held node).
__global__ void coarsest_apply(int n, const double *__restrict__ inv, const uint8_t *__restrict__ active,
                               const double *b, double *x, const CycleIo *__restrict__ io) {
    const int r = threadIdx.x;
    if (r >= n) return;
    if (io) {
        b = io->b;
        x = io->z;
    }
    double s = 0.0;
    for (int c = 0; c < n; ++c) s += inv[r * n + c] * b[c];
    x[r] = active[r] ? s : 0.0;
}

// The 9-point form of the 5-point level-0 operator, for a mesh whose first level is
// already the coarsest (the dense inverse reads 9-point rows).
__global__ void five_to_nine(i64 n, const double *__restrict__ c4, const double *__restrict__ diag,
                             const uint8_t *__restrict__ active, double *__restrict__ a9) {
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n) return;
    for (int q = 0; q < 9; ++q) a9[(i64)q * n + f] = 0.0;
    if (!active[f]) {
        a9[4 * n + f] = 1.0;
        return;
    }
    // place (dI + 1) 3 + (dJ + 1), as every 9-point reader has it
    a9[4 * n + f] = diag[f];
    a9[1 * n + f] = -c4[f];          // (-1, 0)
    a9[7 * n + f] = -c4[n + f];      // (+1, 0)
    a9[3 * n + f] = -c4[2 * n + f];  // (0, -1)
    a9[5 * n + f] = -c4[3 * n + f];  // (0, +1)
}

// -- the small levels in one launch, in shared memory ---------------------------------------

constexpr int kTailThreads = 512;
constexpr int kTailRows = 2;  // rows of the inverse a warp applies at a time
constexpr int kTailMaxLevels = 16;
constexpr size_t kTailSmemMax = 200 * 1024;

struct TailLevel {
    i64 nx, ny, n;
    const double *a9, *rdiag;
    const uint8_t *active;
    double *x, *b;  // the level's global vectors (read: b of the first, written: x of the first)
};

// Where a tail level lives in shared memory.  The block's shared memory is a static image
// -- the levels' coefficients and transfer weights (doubles), transfer indices (int32s) and
// active flags (bytes), copied in one piece from a device buffer kept in step with the
// hierarchy -- then the levels' x (with a ring of zeros), b and r (doubles).  a9, wx, wy,
// rxw, ryw count doubles from the start; lox, loy, rx0, ry0 int32s from the int block; act
// bytes from the byte block; x, b, r doubles from the dynamic block.
struct TailPlan {
    int nx, ny, n, ncx, ncy;
    int x, b, r, a9, rd;     // x: (nx + 2) (ny + 2) with a ring of zeros; b, r: n; a9: 9 n; the
                             // reciprocal diagonal: n
    int wx, wy, rxw, ryw;    // transfer weights to the next level
    int lox, loy, rx0, ry0;  // transfer indices (ints)
    int act;                 // active flags (bytes)
};

struct TailLayout {
    std::vector<TailPlan> plan;
    int doubles = 0, ints = 0, bytes = 0, dynamic = 0;
    // the static image's bytes, rounded up to whole 16-byte words, and where the dynamic
    // doubles start
    size_t image() const {
        const size_t b = sizeof(double) * (size_t)doubles + sizeof(int32_t) * (size_t)ints + bytes;
        return (b + 15) & ~(size_t)15;
    }
    size_t total() const { return image() + sizeof(double) * (size_t)dynamic; }
};

// A thread's place among the nodes of a colour of a level: rows and columns of the even and
// the odd columns' lists, found once for all of a level's phases.
struct TailPlace {
    int row[2], col[2];
};
__device__ __forceinline__ TailPlace tail_place(const TailPlan &P, int tid) {
    TailPlace T;
#pragma unroll
    for (int cj = 0; cj < 2; ++cj) {
        const int hy = (P.ny - cj + 1) >> 1;
        T.row[cj] = tid / hy;
        T.col[cj] = tid - T.row[cj] * hy;
    }
    return T;
}

template <bool PLAIN>
__device__ __forceinline__ void tail_smooth(const TailPlan &P, const TailPlace &T, const double *sm,
                                            double *smd, const uint8_t *act, int colour, int tid,
                                            int nt) {
    const int nx = P.nx, ny = P.ny, n = P.n, W = ny + 2;
    const int ci = colour >> 1, cj = colour & 1;
    const int hx = (nx - ci + 1) >> 1, hy = (ny - cj + 1) >> 1;
    double *x = smd + P.x;
    const double *b = smd + P.b, *a9 = sm + P.a9, *rd = PLAIN ? a9 + 4 * n : sm + P.rd;
    int ti = cj ? T.row[1] : T.row[0], tj = cj ? T.col[1] : T.col[0];
    for (int t = tid; t < hx * hy; t += nt) {
        if (t != tid) {
            ti = t / hy;
            tj = t - ti * hy;
        }
        const int i = 2 * ti + ci, j = 2 * tj + cj;
        const int f = i * ny + j;
        if (!act[f]) continue;
        const int q = (i + 1) * W + j + 1;
        const double c[8] = {a9[f],         a9[n + f],     a9[2 * n + f], a9[3 * n + f],
                             a9[5 * n + f], a9[6 * n + f], a9[7 * n + f], a9[8 * n + f]};
        const double v[8] = {x[q - W - 1], x[q - W],     x[q - W + 1], x[q - 1],
                             x[q + 1],     x[q + W - 1], x[q + W],     x[q + W + 1]};
        x[q] = update9<PLAIN>(b[f], c, v, rd[f]);
    }
}

__device__ __forceinline__ void tail_residual(const TailPlan &P, const double *sm, double *smd,
                                              const uint8_t *act, int tid, int nt) {
    const int ny = P.ny, n = P.n, W = ny + 2;
    const double *x = smd + P.x, *b = smd + P.b, *a9 = sm + P.a9;
    double *r = smd + P.r;
    for (int f = tid; f < n; f += nt) {
        if (!act[f]) {
            r[f] = 0.0;
            continue;
        }
        const int i = f / ny;
        const int q = f + 2 * i + W + 1;
        double s = b[f];
        s -= a9[f] * x[q - W - 1];
        s -= a9[n + f] * x[q - W];
        s -= a9[2 * n + f] * x[q - W + 1];
        s -= a9[3 * n + f] * x[q - 1];
        s -= a9[4 * n + f] * x[q];
        s -= a9[5 * n + f] * x[q + 1];
        s -= a9[6 * n + f] * x[q + W - 1];
        s -= a9[7 * n + f] * x[q + W];
        s -= a9[8 * n + f] * x[q + W + 1];
        r[f] = s;
    }
}

// b of the next level = R r of this one (the next level's x is zero already).
__device__ __forceinline__ void tail_restrict(const TailPlan &P, const TailPlan &C,
                                              const double *sm, double *smd, const int32_t *smi,
                                              const uint8_t *act, int tid, int nt) {
    const int ny = P.ny, ncy = P.ncy;
    const double *r = smd + P.r, *rxw = sm + P.rxw, *ryw = sm + P.ryw;
    const int32_t *rx0 = smi + P.rx0, *ry0 = smi + P.ry0;
    double *bc = smd + C.b;
    for (int t = tid; t < C.n; t += nt) {
        const int I = t / ncy, J = t - I * ncy;
        const int k0 = rx0[I], l0 = ry0[J];
        double s = 0.0;
#pragma unroll
        for (int a = 0; a < kRestrict; ++a) {
            const double px = rxw[kRestrict * I + a];
            if (px == 0.0) continue;
#pragma unroll
            for (int c = 0; c < kRestrict; ++c) {
                const double py = ryw[kRestrict * J + c];
                if (py == 0.0) continue;
                const int f = (k0 + a) * ny + l0 + c;
                if (!act[f]) continue;
                s += px * py * 1.0 * r[f];
            }
        }
        bc[t] = s;
    }
}

// x of this level += P x of the next level.
__device__ __forceinline__ void tail_prolong(const TailPlan &P, const TailPlan &C,
                                             const double *sm, double *smd, const int32_t *smi,
                                             const uint8_t *act, int tid, int nt) {
    const int ny = P.ny, n = P.n, W = ny + 2, ncx = P.ncx, ncy = P.ncy, Wc = ncy + 2;
    double *x = smd + P.x;
    const double *xc = smd + C.x, *wxs = sm + P.wx, *wys = sm + P.wy;
    const int32_t *lox = smi + P.lox, *loy = smi + P.loy;
    for (int f = tid; f < n; f += nt) {
        if (!act[f]) continue;
        const int k = f / ny, l = f - k * ny;
        const int ix = lox[k], iy = loy[l];
        const double wx = wxs[k], wy = wys[l];
        double s = 0.0;
        for (int sx = 0; sx < 2; ++sx) {
            const double px = sx ? 1.0 - wx : wx;
            if (px == 0.0 || ix + sx >= ncx) continue;
            for (int sy = 0; sy < 2; ++sy) {
                const double py = sy ? 1.0 - wy : wy;
                if (py == 0.0 || iy + sy >= ncy) continue;
                s += px * py * xc[(ix + sx + 1) * Wc + iy + sy + 1];
            }
        }
        const int q = f + 2 * k + W + 1;
        x[q] = x[q] + s;
    }
}

// The tail's first level in registers: a thread has one node of each colour, its row, b and
// place in x's layout.  Read from shared memory instead, a phase of 180 nodes was 18 strided
// loads a thread and took 1,175 cycles; 465 so.
struct TailRegisters {
    double coef[4][8], diag[4], rd[4], b[4];
    int at[4], node[4];  // node -1: none, or a held one
};

__device__ __forceinline__ void tail_load(const TailLevel &L, TailRegisters &R, int tid) {
    const int nx = (int)L.nx, ny = (int)L.ny, W = ny + 2;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int ci = k >> 1, cj = k & 1;
        const int hx = (nx - ci + 1) >> 1, hy = (ny - cj + 1) >> 1;
        const int ti = tid / hy, tj = tid - ti * hy;
        const int i = 2 * ti + ci, j = 2 * tj + cj;
        const bool in = tid < hx * hy;
        const int f = in ? i * ny + j : 0;
        const bool on = in && L.active[f] != 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) R.coef[k][q] = L.a9[(i64)(q < 4 ? q : q + 1) * L.n + f];
        R.diag[k] = L.a9[4 * L.n + f];
        R.rd[k] = L.rdiag[f];
        R.b[k] = L.b[f];
        R.at[k] = in ? (i + 1) * W + j + 1 : W + 1;
        R.node[k] = on ? f : (in ? -2 - f : -1);  // -2 - f: held
    }
}

// The eight neighbours of place q in x.
__device__ __forceinline__ void tail_neighbours(const double *x, int W, double (&v)[8]) {
    v[0] = x[-W - 1];
    v[1] = x[-W];
    v[2] = x[-W + 1];
    v[3] = x[-1];
    v[4] = x[1];
    v[5] = x[W - 1];
    v[6] = x[W];
    v[7] = x[W + 1];
}

// A block's number in its cluster, a store to a shared variable of block `rank` of it, and the
// cluster's barrier (which completes such stores) in two halves, of which every thread takes
// the one and the other in turn; a warp's lanes take them together.
__device__ __forceinline__ int cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}
__device__ __forceinline__ void remote_store(const double *p, int rank, double v) {
    uint32_t at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;"
        : "=r"(at)
        : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    cluster_arrive();
    cluster_wait();
}

// The coarsest level's inverse is applied by the other seven blocks of the tail's cluster,
// their rows of it in registers from the launch on: one block alone read the inverse's 346 KB
// (208 nodes) at 20 bytes a cycle, 18,000 of the tail's 39,000 cycles.  The first block sends
// every helper b, the helpers send it x; a barrier each.  A block's shared memory may be
// stored to only once the block has started: every block arrives at a barrier as it starts,
// and the first waits there just before it sends (the helpers once their rows are asked for),
// by when the others have long arrived.
constexpr int kTailCluster = 8;
constexpr int kHelperRows = 3;  // rows a helper's warp: 256 / 7 blocks / 16 warps, rounded up

__device__ __forceinline__ void tail_helper(const TailLevel &L, const TailPlan &C,
                                            const double *__restrict__ inv, double *smd, int rank) {
    const int n = C.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps = kTailThreads / 32 * (kTailCluster - 1);
    const int first = (rank - 1) * (kTailThreads / 32) + warp;  // rows first, first + warps, ..
    constexpr int kChunks = kCoarsest / 32;
    double m[kHelperRows][kChunks];
    bool on[kHelperRows];
#pragma unroll
    for (int k = 0; k < kHelperRows; ++k) {
        const int row = first + k * warps;
        on[k] = row < n && L.active[row] != 0;
#pragma unroll
        for (int e = 0; e < kChunks; ++e) {
            const int c = lane + 32 * e;
            m[k][e] = row < n && c < n ? __ldg(inv + (i64)row * n + c) : 0.0;
        }
    }
    cluster_wait();     // (of the start's barrier)
    cluster_barrier();  // b is here
    const double *b = smd + C.b;
#pragma unroll
    for (int k = 0; k < kHelperRows; ++k) {
        const int row = first + k * warps;
        double s = 0.0;
#pragma unroll
        for (int e = 0; e < kChunks; ++e)
            s = fma(m[k][e], lane + 32 * e < n ? b[lane + 32 * e] : 0.0, s);
        for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
        if (lane == 0 && row < n)
            remote_store(smd + C.x + row + 2 * (row / C.ny) + C.ny + 3, 0, on[k] ? s : 0.0);
    }
    cluster_barrier();  // x is there
}

// levels[0] reads b from, and writes x to, global memory; `image` holds the static part
// of the shared memory (image_words 16-byte words); inv is the coarsest level's inverse.
// The first block of a cluster, whose other blocks are tail_helpers; PLAIN: a batch's, in its
// arithmetic (update9), one block a candidate.
// (The body of vcycle_tail and of batch_tail.)
template <bool PLAIN>
__device__ __forceinline__ void vcycle_tail_run(const TailLevel *__restrict__ levels,
                                                const TailPlan *__restrict__ plans, int count,
                                                const uint4 *__restrict__ image,
                                                int image_words, int doubles, int ints,
                                                const double *__restrict__ inv, int sweeps) {
    extern __shared__ __align__(16) double sm[];
    __shared__ TailPlan plan[kTailMaxLevels];
    int32_t *smi = reinterpret_cast<int32_t *>(sm + doubles);
    uint8_t *smb = reinterpret_cast<uint8_t *>(smi + ints);
    double *smd = sm + 2 * image_words;  // the dynamic doubles follow the image
    const int tid = threadIdx.x, nt = blockDim.x;
    if (!PLAIN) {
        cluster_arrive();  // this block has started
        const int rank = cluster_rank();
        if (rank != 0) {
            tail_helper(levels[count - 1], plans[count - 1], inv, smd, rank);
            return;
        }
    }
    TailRegisters R;
    if (count > 1) tail_load(levels[0], R, tid);
    {
        const int *src = reinterpret_cast<const int *>(plans);
        int *dst = reinterpret_cast<int *>(plan);
        const int words = count * (int)(sizeof(TailPlan) / sizeof(int));
        for (int e = tid; e < words; e += nt) dst[e] = src[e];
    }
    // the static image in one piece (its first doubles are the first level's ten coefficients
    // a node, held in registers), x zero, level 0's b
    uint4 *dst = reinterpret_cast<uint4 *>(sm);
    const int skip = count > 1 ? 5 * plans[0].n : 0;
#pragma unroll 4
    for (int e = skip + tid; e < image_words; e += nt) dst[e] = image[e];
    for (int l = 0; l < count; ++l) {
        const TailPlan &P = plans[l];
        for (int e = tid; e < (P.nx + 2) * (P.ny + 2); e += nt) smd[P.x + e] = 0.0;
    }
    if (count == 1) {
        const TailPlan &P = plans[0];
        const double *b0 = levels[0].b;
        for (int f = tid; f < P.n; f += nt) smd[P.b + f] = b0[f];
    }
    __syncthreads();
    // one colour phase of the first level
    auto phase = [&](double *x, int W, int k) {
        if (R.node[k] >= 0) {
            double v[8];
            tail_neighbours(x + R.at[k], W, v);
            x[R.at[k]] = update9<PLAIN>(R.b[k], R.coef[k], v, PLAIN ? R.diag[k] : R.rd[k]);
        }
        __syncthreads();
    };
    for (int l = 0; l + 1 < count; ++l) {
        const TailPlan &P = plan[l];
        const uint8_t *act = smb + P.act;
        if (l == 0) {
            double *x = smd + P.x, *r = smd + P.r;
            const int W = P.ny + 2;
            for (int s = 0; s < sweeps; ++s) {
#pragma unroll
                for (int c = 0; c < 4; ++c) phase(x, W, c);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (R.node[k] >= 0) {
                    double v[8];
                    tail_neighbours(x + R.at[k], W, v);
                    if (PLAIN) {
                        double p = R.b[k];
#pragma unroll
                        for (int e = 0; e < 4; ++e) p -= R.coef[k][e] * v[e];
                        p -= R.diag[k] * x[R.at[k]];
#pragma unroll
                        for (int e = 4; e < 8; ++e) p -= R.coef[k][e] * v[e];
                        r[R.node[k]] = p;
                    } else {
                        double p = fma(-R.diag[k], x[R.at[k]], R.b[k]), q = R.coef[k][7] * v[7];
#pragma unroll
                        for (int e = 0; e < 4; ++e) p = fma(-R.coef[k][e], v[e], p);
#pragma unroll
                        for (int e = 4; e < 7; ++e) q = fma(R.coef[k][e], v[e], q);
                        r[R.node[k]] = p - q;
                    }
                } else if (R.node[k] <= -2) {
                    r[-2 - R.node[k]] = 0.0;
                }
            }
        } else {
            const TailPlace T = tail_place(P, tid);
            for (int s = 0; s < sweeps; ++s)
                for (int c = 0; c < 4; ++c) {
                    tail_smooth<PLAIN>(P, T, sm, smd, act, c, tid, nt);
                    __syncthreads();
                }
            tail_residual(P, sm, smd, act, tid, nt);
        }
        __syncthreads();
        tail_restrict(P, plan[l + 1], sm, smd, smi, act, tid, nt);
        __syncthreads();
    }
    if (!PLAIN) {
        const TailPlan &C = plan[count - 1];
        cluster_wait();  // every helper has started
        for (int e = tid; e < C.n * (kTailCluster - 1); e += nt) {
            const int rank = 1 + e / C.n, f = e - (rank - 1) * C.n;
            remote_store(smd + C.b + f, rank, smd[C.b + f]);
        }
        cluster_barrier();
        cluster_barrier();
    } else {
        // the coarsest level: x = inv b, a warp kTailRows rows at a time, its lanes over the
        // columns
        const TailPlan &C = plan[count - 1];
        const int n = C.n, W = C.ny + 2, lane = tid & 31, warps = nt >> 5;
        const double *b = smd + C.b;
        const uint8_t *act = smb + C.act;
        constexpr int kChunks = kCoarsest / 32;
        for (int row = tid >> 5; row < n; row += kTailRows * warps) {
            double s[kTailRows], m[kTailRows][kChunks];
#pragma unroll
            for (int e = 0; e < kChunks; ++e) {
                const int c = lane + 32 * e;
#pragma unroll
                for (int k = 0; k < kTailRows; ++k)
                    m[k][e] = c < n && row + k * warps < n
                                  ? __ldg(inv + (i64)(row + k * warps) * n + c) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < kTailRows; ++k) s[k] = 0.0;
#pragma unroll
            for (int e = 0; e < kChunks; ++e) {
                const double v = lane + 32 * e < n ? b[lane + 32 * e] : 0.0;
#pragma unroll
                for (int k = 0; k < kTailRows; ++k)
                    s[k] = s[k] + m[k][e] * v;
            }
            for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
                for (int k = 0; k < kTailRows; ++k) s[k] += __shfl_down_sync(0xffffffffu, s[k], off);
            }
            if (lane == 0) {
#pragma unroll
                for (int k = 0; k < kTailRows; ++k) {
                    const int r = row + k * warps;
                    if (r < n) smd[C.x + r + 2 * (r / C.ny) + W + 1] = act[r] ? s[k] : 0.0;
                }
            }
        }
        __syncthreads();
    }
    for (int l = count - 2; l >= 0; --l) {
        const TailPlan &P = plan[l];
        const uint8_t *act = smb + P.act;
        tail_prolong(P, plan[l + 1], sm, smd, smi, act, tid, nt);
        __syncthreads();
        if (l == 0) {
            double *x = smd + P.x;
            for (int s = 0; s < sweeps; ++s) {
#pragma unroll
                for (int c = 3; c >= 0; --c) phase(x, P.ny + 2, c);
            }
        } else {
            const TailPlace T = tail_place(P, tid);
            for (int s = 0; s < sweeps; ++s)
                for (int c = 3; c >= 0; --c) {
                    tail_smooth<PLAIN>(P, T, sm, smd, act, c, tid, nt);
                    __syncthreads();
                }
        }
    }
    {
        const TailPlan &P = plan[0];
        const int W = P.ny + 2;
        double *x0 = levels[0].x;
        for (int f = tid; f < P.n; f += nt) x0[f] = smd[P.x + f + 2 * (f / P.ny) + W + 1];
    }
}

__global__ void __launch_bounds__(kTailThreads, 1) __cluster_dims__(kTailCluster, 1, 1)
    vcycle_tail(const TailLevel *__restrict__ levels, const TailPlan *__restrict__ plans, int count,
                const uint4 *__restrict__ image, int image_words, int doubles, int ints,
                const double *__restrict__ inv, int sweeps) {
    vcycle_tail_run<false>(levels, plans, count, image, image_words, doubles, ints, inv, sweeps);
}

// Whether a colour of a tail's first level fits the block's threads, which hold it in
// registers: no level with more nodes of a colour fits the shared memory (the smallest such
// takes 260 KB), so this ends no tail earlier than that does.
bool tail_fits_threads(i64 nx, i64 ny) { return ((nx + 1) / 2) * ((ny + 1) / 2) <= kTailThreads; }

// The shared-memory layout of tail levels first .. (the coarsest): the static image
// (coefficients of every level but the coarsest, transfer tables, active flags), then the
// dynamic x, b, r of every level.
TailLayout tail_layout(const std::vector<Level> &levels, int first) {
    TailLayout T;
    const int last = (int)levels.size() - 1;
    for (int l = first; l <= last; ++l) {
        const Level &L = levels[l];
        TailPlan P{};
        P.nx = (int)L.nx;
        P.ny = (int)L.ny;
        P.n = (int)L.n;
        if (l < last) {
            P.ncx = (int)levels[l + 1].nx;
            P.ncy = (int)levels[l + 1].ny;
            P.a9 = T.doubles;
            T.doubles += 9 * P.n;
            P.rd = T.doubles;
            T.doubles += P.n;
            P.wx = T.doubles;
            T.doubles += P.nx;
            P.wy = T.doubles;
            T.doubles += P.ny;
            P.rxw = T.doubles;
            T.doubles += kRestrict * P.ncx;
            P.ryw = T.doubles;
            T.doubles += kRestrict * P.ncy;
            P.lox = T.ints;
            T.ints += P.nx;
            P.loy = T.ints;
            T.ints += P.ny;
            P.rx0 = T.ints;
            T.ints += P.ncx;
            P.ry0 = T.ints;
            T.ints += P.ncy;
        }
        P.act = T.bytes;
        T.bytes += P.n;
        P.x = T.dynamic;
        T.dynamic += (P.nx + 2) * (P.ny + 2);
        P.b = T.dynamic;
        T.dynamic += P.n;
        P.r = T.dynamic;
        T.dynamic += P.n;
        T.plan.push_back(P);
    }
    return T;
}

// -- sums over a vector: partial sums per block, the last block adds them in block order ----

constexpr int kDotMax = 32;       // at most this many vectors against one
constexpr int kDotBlocks = 148;   // one per SM, of at least an element a thread
constexpr int kDotThreads = 512;

int dot_blocks(i64 n) { return (int)std::min<i64>(kDotBlocks, (n + kDotThreads - 1) / kDotThreads); }

// out[q] = the sum of every thread's acc[q], q < sums <= NACC: the threads of a warp, the warps
// of a block and the blocks are added in a fixed order, the blocks' partials by the block
// that finishes last (a ticket counter, reset by it): the same bits on every run, in one
// launch.  True in the last block, whose threads may then read `out` (after its barrier).
template <int NACC>
__device__ __forceinline__ bool grid_sums(const double (&acc)[NACC], int sums,
                                          double *__restrict__ partial,
                                          unsigned *__restrict__ ticket, double *out) {
    constexpr int kWarps = kDotThreads / 32;
    __shared__ double warp_part[kWarps][NACC];
    __shared__ bool is_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NACC; ++q) {
        if (q >= sums) break;
        double v = acc[q];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) warp_part[warp][q] = v;
    }
    __syncthreads();
    if (threadIdx.x < sums) {
        double v = 0.0;
#pragma unroll
        for (int wi = 0; wi < kWarps; ++wi) v += warp_part[wi][threadIdx.x];
        partial[(i64)blockIdx.x * kDotMax + threadIdx.x] = v;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!is_last) return false;
    __threadfence();
    // a warp a sum: its lanes read the blocks' partials together, then add them
    constexpr int kPer = (kDotBlocks + 31) / 32;
    const int blocks = (int)gridDim.x;
    for (int q = warp; q < sums; q += kWarps) {
        double part[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int b = lane + 32 * k;
            part[k] = b < blocks ? __ldcg(partial + (i64)b * kDotMax + q) : 0.0;
        }
        double v = 0.0;
#pragma unroll
        for (int k = 0; k < kPer; ++k)
            if (lane + 32 * k < blocks) v += part[k];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) out[q] = v;
    }
    if (threadIdx.x == 0) *ticket = 0u;
    __syncthreads();
    return true;
}

// -- vector kernels of GMRES and Newton ----------------------------------------------------

// The Arnoldi process of one GMRES restart cycle, on the device: the Hessenberg matrix H
// ((m + 1) x m, row-major), the Givens rotations (cs, sn) and the rotated right-hand side
// g.  `j` counts the steps taken; once `done` (the residual estimate |g[j]| at the
// tolerance, or a breakdown) later steps change nothing, so the host may queue steps past
// the end and the cycle's solution is the same.
struct Arnoldi {
    int j, done;
    double tol;
    double resid[kDotMax + 1];  // |g[j]| after step j
};

__global__ void set_cycle(CycleIo *__restrict__ io, const double *b, double *z) {
    io->b = b;
    io->z = z;
}

__global__ void cycle_begin(const CycleIo *__restrict__ io, i64 n, double *__restrict__ b,
                            double *__restrict__ x) {
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n) return;
    b[f] = io->b[f];
    x[f] = 0.0;
}

__global__ void cycle_end(const CycleIo *__restrict__ io, i64 n, const double *__restrict__ x) {
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f < n) io->z[f] = x[f];
}

// A cycle begins: V_0 = r / beta, the state empty, the V-cycle's vectors the first.
__global__ void arnoldi_begin(Arnoldi *__restrict__ a, double *__restrict__ g, int m, double beta,
                              double tol, const double *__restrict__ r, i64 n,
                              double *__restrict__ V, double *__restrict__ Z,
                              CycleIo *__restrict__ io) {
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f < n) V[f] = (1.0 / beta) * r[f];
    if (f != 0) return;
    a->j = 0;
    a->done = 0;
    a->tol = tol;
    a->resid[0] = beta;
    g[0] = beta;
    for (int q = 1; q <= m; ++q) g[q] = 0.0;
    io->b = V;
    io->z = Z;
}

// Step j: the new Hessenberg column from the two Gram-Schmidt passes' coefficients h1, h2
// and the new vector's squared norm, rotated by the earlier rotations; the new rotation and
// g, whose last entry is the residual norm up to its sign.  A block's first warp.
__device__ __forceinline__ void arnoldi_step(Arnoldi *__restrict__ a, double *__restrict__ H,
                                             double *__restrict__ cs, double *__restrict__ sn,
                                             double *__restrict__ g, const double *__restrict__ h1,
                                             const double *__restrict__ h2, const double *norm2,
                                             int j, int m) {
    // the warp reads the column's coefficients and the rotations together; one thread then
    // rotates the column in shared memory and writes it out
    __shared__ double col[kDotMax + 2], c[kDotMax], sv[kDotMax];
    const int t = threadIdx.x;
    if (t >= 32 || a->done || a->j != j) return;
    for (int q = t; q <= j; q += 32) col[q] = h1[q] + h2[q];
    for (int q = t; q < j; q += 32) {
        c[q] = cs[q];
        sv[q] = sn[q];
    }
    __syncwarp();
    if (t != 0) return;
    const double hn = sqrt(norm2[0]);
    col[j + 1] = hn;
    for (int q = 0; q < j; ++q) {
        const double x = col[q], y = col[q + 1];
        col[q] = c[q] * x + sv[q] * y;
        col[q + 1] = -sv[q] * x + c[q] * y;
    }
    const double x = col[j], y = col[j + 1];
    const double rr = hypot(x, y);
    const double cj = rr > 0.0 ? x / rr : 1.0;
    const double sj = rr > 0.0 ? y / rr : 0.0;
    col[j] = rr;
    col[j + 1] = 0.0;
    for (int q = 0; q <= j + 1; ++q) H[q * m + j] = col[q];
    cs[j] = cj;
    sn[j] = sj;
    const double gj = g[j];
    g[j + 1] = -sj * gj;
    g[j] = cj * gj;
    a->j = j + 1;
    a->resid[j + 1] = fabs(g[j + 1]);
    if (fabs(g[j + 1]) <= a->tol || hn == 0.0) a->done = 1;
}

// The rows of the finest operator, for the kernels that apply it as they go.
struct Rows5 {
    i64 nx, ny;
    const double *c4, *diag;
    const uint8_t *active;
};

__device__ __forceinline__ double apply_row(const Rows5 &A, i64 f, const double *__restrict__ x) {
    if (!A.active[f]) return 0.0;
    const i64 n = A.nx * A.ny;
    const int ny = (int)A.ny, i = (int)((unsigned)f / (unsigned)ny), j = (int)f - i * ny;
    double s = A.diag[f] * x[f];
    if (i > 0) s -= A.c4[f] * x[f - ny];
    if (i < (int)A.nx - 1) s -= A.c4[n + f] * x[f + ny];
    if (j > 0) s -= A.c4[2 * n + f] * x[f - 1];
    if (j < ny - 1) s -= A.c4[3 * n + f] * x[f + 1];
    return s;
}

// A Krylov step's three passes over the new vector w and the basis V (m = j + 1 rows):
// kApply: w = A z and h1[q] = <V_q, w>; kOrthDots: w -= sum_q h1[q] V_q (classical
// Gram-Schmidt) and h2[q] = <V_q, w>; kOrthNorm: w -= sum_q h2[q] V_q, its squared norm, and in
// the last block the step's Hessenberg column and rotation (arnoldi_step).  Three launches and
// the scaling of the next basis vector, where the product, three passes, the scaling, the
// column and the V-cycle's copies in and out took nine: 9 to 13 us a pass at 801 x 201.
enum PassMode { kApply = 0, kOrthDots = 1, kOrthNorm = 2 };

struct ArnoldiState {
    Arnoldi *a;
    double *H, *cs, *sn, *g, *h1, *h2, *hn;
    int j, m;  // the step and the cycle's length
};

template <int MQ, int MODE>
__global__ void __launch_bounds__(kDotThreads) krylov_pass(
    Rows5 A, const double *__restrict__ V, const double *__restrict__ z, double *w, i64 n, int m,
    ArnoldiState S, double *__restrict__ partial, unsigned *__restrict__ ticket) {
    constexpr int NACC = MODE == kOrthNorm ? 1 : MQ;
    double acc[NACC];
#pragma unroll
    for (int q = 0; q < NACC; ++q) acc[q] = 0.0;
    const double *h = MODE == kOrthNorm ? S.h2 : S.h1;
    for (i64 f = (i64)blockIdx.x * kDotThreads + threadIdx.x; f < n;
         f += (i64)gridDim.x * kDotThreads) {
        double vq[MQ];
#pragma unroll
        for (int q = 0; q < MQ; ++q)
            if (q < m) vq[q] = V[(i64)q * n + f];
        double s;
        if (MODE == kApply) {
            s = apply_row(A, f, z);
        } else {
            s = w[f];
#pragma unroll
            for (int q = 0; q < MQ; ++q)
                if (q < m) s -= h[q] * vq[q];
        }
        w[f] = s;
        if (MODE == kOrthNorm) {
            acc[0] += s * s;
        } else {
#pragma unroll
            for (int q = 0; q < MQ; ++q)
                if (q < m) acc[q] += vq[q] * s;
        }
    }
    double *out = MODE == kApply ? S.h1 : (MODE == kOrthDots ? S.h2 : S.hn);
    const bool last = grid_sums(acc, MODE == kOrthNorm ? 1 : m, partial, ticket, out);
    if (MODE == kOrthNorm && last)
        arnoldi_step(S.a, S.H, S.cs, S.sn, S.g, S.h1, S.h2, S.hn, S.j, S.m);
}

// out[0] = |u|^2, out[1] = |r|^2 of r = u - A x (r also written)
__global__ void __launch_bounds__(kDotThreads) residual_norms(Rows5 A, const double *__restrict__ u,
                                                              const double *__restrict__ x, i64 n,
                                                              double *__restrict__ r,
                                                              double *__restrict__ partial,
                                                              unsigned *__restrict__ ticket,
                                                              double *__restrict__ out) {
    double acc[2] = {0.0, 0.0};
    for (i64 f = (i64)blockIdx.x * kDotThreads + threadIdx.x; f < n;
         f += (i64)gridDim.x * kDotThreads) {
        const double b = u[f], v = A.active[f] ? b - apply_row(A, f, x) : 0.0;
        r[f] = v;
        acc[0] += b * b;
        acc[1] += v * v;
    }
    grid_sums(acc, 2, partial, ticket, out);
}

// out[0] = |v|^2
__global__ void __launch_bounds__(kDotThreads) vector_norm(const double *__restrict__ v, i64 n,
                                                           double *__restrict__ partial,
                                                           unsigned *__restrict__ ticket,
                                                           double *__restrict__ out) {
    double acc[1] = {0.0};
    for (i64 f = (i64)blockIdx.x * kDotThreads + threadIdx.x; f < n;
         f += (i64)gridDim.x * kDotThreads)
        acc[0] += v[f] * v[f];
    grid_sums(acc, 1, partial, ticket, out);
}

// y = H^-1 g on the leading j x j upper triangle (j the steps taken)
__global__ void arnoldi_solve(const Arnoldi *__restrict__ a, const double *__restrict__ H,
                              const double *__restrict__ g, double *__restrict__ y, int m) {
    if (threadIdx.x != 0) return;
    const int j = a->j;
    for (int q = j - 1; q >= 0; --q) {
        double s = g[q];
        for (int c = q + 1; c < j; ++c) s -= H[q * m + c] * y[c];
        y[q] = s / H[q * m + q];
    }
}

// V_{j+1} = w / sqrt(norm2[0]) (zero for a zero norm: GMRES stops there), the next V-cycle's
// vectors with it.
__global__ void scale_by_norm(const double *__restrict__ w, const double *__restrict__ norm2, i64 n,
                              double *__restrict__ v, double *z, CycleIo *__restrict__ io) {
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f == 0) {
        io->b = v;
        io->z = z;
    }
    if (f >= n) return;
    const double s = norm2[0];
    v[f] = s > 0.0 ? w[f] / sqrt(s) : 0.0;
}

// x += sum_q y[q] Z[q], q below the cycle's steps
__global__ void combine(const double *__restrict__ Z, const double *__restrict__ y,
                        const Arnoldi *__restrict__ a, i64 n, double *__restrict__ x) {
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n) return;
    const int m = a->j;
    double s = x[f];
    for (int q = 0; q < m; ++q) s += y[q] * Z[(i64)q * n + f];
    x[f] = s;
}

// the larger of two values, NaN if either is (a NaN update must not read as converged)
__device__ __forceinline__ double max_nan(double m, double v) {
    return (v > m || v != v) ? v : m;
}

// x += d and *out = max |d| (NaN if any entry is NaN): Newton's update and its size in one
// pass over the vectors.  Every block leaves its maximum, the block that finishes last (a
// ticket counter, reset by it) takes theirs; a maximum does not depend on the order.  One
// block alone took 307 us for 525,825 nodes; a grid of a block a multiprocessor 9 us
// with the addition.
__global__ void __launch_bounds__(kDotThreads) add_max(const double *__restrict__ d, i64 n,
                                                       double *__restrict__ x,
                                                       double *__restrict__ partial,
                                                       unsigned *__restrict__ ticket,
                                                       double *__restrict__ out) {
    __shared__ double part[kDotThreads / 32];
    __shared__ bool is_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto block_max = [&](double m) {
        for (int off = 16; off > 0; off >>= 1)
            m = max_nan(m, __shfl_down_sync(0xffffffffu, m, off));
        if (lane == 0) part[warp] = m;
        __syncthreads();
        m = part[0];
        for (int w = 1; w < kDotThreads / 32; ++w) m = max_nan(m, part[w]);
        __syncthreads();
        return m;
    };
    double m = 0.0;
    for (i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x; f < n;
         f += (i64)gridDim.x * blockDim.x) {
        const double v = d[f];
        x[f] += v;
        m = max_nan(m, fabs(v));
    }
    m = block_max(m);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = m;
        __threadfence();
        is_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    m = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
        m = max_nan(m, __ldcg(partial + b));
    m = block_max(m);
    if (threadIdx.x == 0) {
        *out = m;
        *ticket = 0u;
    }
}

// the right-hand side: rho / eps0 + c on free nodes, 0 on fixed ones; phi's fixed values set
__global__ void prepare(i64 n, const double *__restrict__ rho, const double *__restrict__ src,
                        const uint8_t *__restrict__ active, const double *__restrict__ value,
                        double *__restrict__ b, double *__restrict__ phi) {
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n) return;
    if (active[f]) {
        b[f] = (rho ? rho[f] / kEps0 : 0.0) + src[f];
    } else {
        b[f] = 0.0;
        phi[f] = value[f];
    }
}

// The Boltzmann species at phi: e = a exp(min(-s (phi - up) / T, 50)); the Newton
// residual r = b + s e - A phi (the negative of F) and the reaction e / T, on free nodes.
__global__ void boltzmann(i64 nx, i64 ny, const double *__restrict__ c4,
                          const double *__restrict__ base, const uint8_t *__restrict__ active,
                          const double *__restrict__ phi, const double *__restrict__ b,
                          double amplitude, double temperature, double up, double sign,
                          double *__restrict__ r, double *__restrict__ reaction) {
    const i64 n = nx * ny;
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n) return;
    if (!active[f]) {
        r[f] = 0.0;
        reaction[f] = 0.0;
        return;
    }
    const i64 i = f / ny, j = f - i * ny;
    double s = base[f] * phi[f];
    if (i > 0) s -= c4[f] * phi[f - ny];
    if (i < nx - 1) s -= c4[n + f] * phi[f + ny];
    if (j > 0) s -= c4[2 * n + f] * phi[f - 1];
    if (j < ny - 1) s -= c4[3 * n + f] * phi[f + 1];
    const double e = amplitude * exp(fmin(-sign * (phi[f] - up) / temperature, 50.0));
    r[f] = b[f] + sign * e - s;
    reaction[f] = e / temperature;
}

__global__ void add_into(const double *__restrict__ d, i64 n, double *__restrict__ x) {
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f < n) x[f] += d[f];
}

void build_axis(Axis &A, i64 n) {
    A.n = n;
    A.coarsened = n > 3;
    A.nc = A.coarsened ? n / 2 + 1 : n;
    std::vector<int32_t> lo(n), cidx(A.nc);
    std::vector<double> w(n);
    for (i64 I = 0; I < A.nc; ++I) cidx[I] = (int32_t)(A.coarsened ? std::min<i64>(2 * I, n - 1) : I);
    for (i64 k = 0; k < n; ++k) {
        if (!A.coarsened) {
            lo[k] = (int32_t)k;
            w[k] = 1.0;
            continue;
        }
        i64 I = std::min<i64>(k / 2, A.nc - 2);
        const double c0 = cidx[I], c1 = cidx[I + 1];
        lo[k] = (int32_t)I;
        w[k] = (c1 - (double)k) / (c1 - c0);
    }
    // the restriction tables: the prolongation weights read by coarse node
    std::vector<int32_t> r0(A.nc, 0);
    std::vector<double> rw((size_t)kRestrict * A.nc, 0.0);
    for (i64 I = 0; I < A.nc; ++I) {
        i64 first = -1;
        for (i64 k = 0; k < n; ++k) {
            const double p = lo[k] == I ? w[k] : (lo[k] + 1 == I ? 1.0 - w[k] : 0.0);
            if (p == 0.0) continue;
            if (first < 0) first = k;
            BT_REQUIRE(k - first < kRestrict, "poisson: a coarse node restricts from too many nodes");
            rw[(size_t)kRestrict * I + (k - first)] = p;
        }
        r0[I] = (int32_t)std::max<i64>(first, 0);
    }
    cudaMemcpy(A.r0.as<int32_t>(A.nc), r0.data(), A.nc * sizeof(int32_t), cudaMemcpyHostToDevice);
    cudaMemcpy(A.rw.as<double>(kRestrict * A.nc), rw.data(), rw.size() * sizeof(double),
               cudaMemcpyHostToDevice);
    cudaMemcpy(A.lo.as<int32_t>(n), lo.data(), n * sizeof(int32_t), cudaMemcpyHostToDevice);
    cudaMemcpy(A.w.as<double>(n), w.data(), n * sizeof(double), cudaMemcpyHostToDevice);
}

}  // namespace
}  // namespace bt

struct bt_poisson {
    bt_ctx *ctx = nullptr;
    i64 nx = 0, ny = 0, n = 0;
    double h = 0.0;
    int cyl = 0;
    i64 j0 = 0;  // the radial index of the first row (origin_y / h; cylindrical)
    double neumann[4] = {0, 0, 0, 0};
    bt::Buffer x, fixed, value, distance, region;  // mesh; region: the extra held nodes
    bt::Buffer fixed_eff, value_eff, src;
    double region_value = 0.0;
    bool has_region = false;
    std::vector<bt::Level> levels;
    bt::Buffer inv, status, band;  // the coarsest inverse; the band's factors
    bool built = false;        // hierarchy matches the current diagonal
    bool transposed = false;   // the fine operator is A's transpose (bt_poisson_set_transposed)
    bt::Buffer c4_plain;       // A's own coefficients while the operator is transposed
    bool reaction_on = false;  // level-0 diagonal holds a reaction
    int restart = 30;
    // the V-cycle's settings (bt_poisson_set_options)
    int fine_sweeps = 2;    // red-black sweeps on level 0, before and after
    int coarse_sweeps = 2;  // four-colour sweeps on the 9-point levels
    int staged = 1;         // smoothing staged through shared memory (else a launch per colour)
    i64 tail_nodes = 4096;  // levels at most this large may go to the one-block tail
    int tail_start = -1;    // the first level of the V-cycle's one-block tail
    size_t tail_smem = 0;   // its shared memory
    int tail_doubles = 0, tail_ints = 0, tail_words = 0;  // its layout (bt::TailLayout)
    bt::Buffer tail_levels;  // its TailLevel descriptors
    bt::Buffer tail_plans;   // and TailPlan layouts
    bt::Buffer tail_image;   // the static part of its shared memory (tail_words 16-byte words)
    bt::Buffer dot_partial;  // per-block partial dot products
    bt::Buffer dot_ticket;   // the dot passes' finishing-block counter (zero between passes)
    bool ticket_ready = false;
    bt::Buffer arnoldi;      // the device Arnoldi state of GMRES (bt::Arnoldi, H, rotations)
    bt::Buffer cycle_io;     // the V-cycle's vectors (bt::CycleIo)
    // the V-cycle from a zero guess on level 0's b into its x, captured once as a graph
    cudaGraph_t vgraph = nullptr;
    cudaGraphExec_t vexec = nullptr;
    i64 vgraph_kernels = 0;
    ~bt_poisson() {
        if (vexec) cudaGraphExecDestroy(vexec);
        if (vgraph) cudaGraphDestroy(vgraph);
    }
    // GMRES: the Krylov basis V, its preconditioned images Z, two work vectors; the solve:
    // its right-hand side, the residual GMRES reduces, the correction, the Newton reaction
    // and scalars.
    bt::Buffer V, Z, work, work2, rhs, r0, delta, reaction, scalars;
};

namespace bt {
namespace {

void refresh_tail_image(bt_poisson *p, bool tables = false);

Fine fine_of(Level &L, Level &C, bool first) {
    Fine F{};
    F.nx = L.nx;
    F.ny = L.ny;
    if (first) {
        F.c4 = L.c4.as<double>(4 * L.n);
        F.diag = L.diag.as<double>(L.n);
        F.a9 = nullptr;
        F.weight = L.weight.as<double>(L.n);
    } else {
        F.c4 = nullptr;
        F.diag = nullptr;
        F.a9 = L.a9.as<double>(9 * L.n);
        F.weight = nullptr;
    }
    F.active = L.active.as<uint8_t>(L.n);
    F.lox = L.ax.lo.as<int32_t>(L.nx);
    F.loy = L.ay.lo.as<int32_t>(L.ny);
    F.wx = L.ax.w.as<double>(L.nx);
    F.wy = L.ay.w.as<double>(L.ny);
    F.rx0 = L.ax.r0.as<int32_t>(L.ax.nc);
    F.ry0 = L.ay.r0.as<int32_t>(L.ay.nc);
    F.rxw = L.ax.rw.as<double>(kRestrict * L.ax.nc);
    F.ryw = L.ay.rw.as<double>(kRestrict * L.ay.nc);
    F.ncx = C.nx;
    F.ncy = C.ny;
    return F;
}

void build_operator(bt_poisson *p) {
    cudaStream_t st = p->ctx->stream;
    Level &L = p->levels[0];
    const i64 n = p->n;
    BT_LAUNCH(p->ctx, build_fine, blocks_for(n, 256), 256, 0, st, p->nx, p->ny, p->x.as<double>(p->nx), p->h, p->cyl, p->j0, p->fixed_eff.as<uint8_t>(n),
        p->distance.as<double>(4 * n), p->neumann[0], p->neumann[1], p->neumann[2],
        p->neumann[3], L.c4.as<double>(4 * n), L.base.as<double>(n), p->src.as<double>(n),
        L.weight.as<double>(n), L.active.as<uint8_t>(n));
    if (p->transposed) {
        double *plain = p->c4_plain.as<double>(4 * n);
        BT_CUDA(cudaMemcpyAsync(plain, L.c4.as<double>(4 * n), sizeof(double) * 4 * n,
                                cudaMemcpyDeviceToDevice, st));
        BT_LAUNCH(p->ctx, transpose_c4, blocks_for(n, 256), 256, 0, st, p->nx, p->ny, plain,
                  L.weight.as<double>(n), L.active.as<uint8_t>(n), L.c4.as<double>(4 * n));
    }
    BT_CHECK_LAUNCH();
    p->built = false;
    p->reaction_on = true;  // force the diagonal to be set
}

// The coarse operators of the hierarchy, and the banded factors and inverse of the coarsest.
template <bool PLAIN>
void coarse_operators(bt_poisson *p) {
    cudaStream_t st = p->ctx->stream;
    for (size_t l = 0; l + 1 < p->levels.size(); ++l) {
        Level &L = p->levels[l], &C = p->levels[l + 1];
        Fine F = fine_of(L, C, l == 0);
        const unsigned grid = blocks_for(C.n, kGalerkinThreads);
        if (F.a9)
            BT_LAUNCH(p->ctx, (galerkin<true, PLAIN>), grid, kGalerkinThreads, 0, st, F,
                      C.a9.as<double>(9 * C.n), C.rdiag.as<double>(C.n), C.active.as<uint8_t>(C.n));
        else
            BT_LAUNCH(p->ctx, (galerkin<false, PLAIN>), grid, kGalerkinThreads, 0, st, F,
                      C.a9.as<double>(9 * C.n), C.rdiag.as<double>(C.n), C.active.as<uint8_t>(C.n));
    }
}
template <bool PLAIN>
void coarsest_band(bt_poisson *p, const double *a9c, double *inv, int *status) {
    cudaStream_t st = p->ctx->stream;
    const Level &Lc = p->levels.back();
    const int nx = (int)Lc.nx, ny = (int)Lc.ny, n = nx * ny, b = band_half(nx, ny);
    double *factors = p->band.as<double>((size_t)n * (2 * kBandPad + 1));
    BT_LAUNCH(p->ctx, coarsest_band_factor<PLAIN>, 1, 32 * b, band_smem(nx, ny), st, nx, ny, a9c,
              factors, status + 1);
    const unsigned grid = blocks_for(n, kSolveThreads);
    const auto smem = [&](int kb) { return sizeof(double) * (size_t)n * (2 * kb + 1); };
    if (b <= 6)
        BT_LAUNCH(p->ctx, (coarsest_band_solve<6, PLAIN>), grid, kSolveThreads, smem(6), st, nx, ny,
                  factors, inv, status + 1);
    else if (b <= 10)
        BT_LAUNCH(p->ctx, (coarsest_band_solve<10, PLAIN>), grid, kSolveThreads, smem(10), st, nx, ny,
                  factors, inv, status + 1);
    else if (b <= 14)
        BT_LAUNCH(p->ctx, (coarsest_band_solve<14, PLAIN>), grid, kSolveThreads, smem(14), st, nx, ny,
                  factors, inv, status + 1);
    else
        BT_LAUNCH(p->ctx, (coarsest_band_solve<18, PLAIN>), grid, kSolveThreads, smem(18), st, nx, ny,
                  factors, inv, status + 1);
}

// Set the level-0 diagonal (with `reaction`, or without) and rebuild the coarse levels.  A
// batch takes single solvers' operators without a reaction, so those are PLAIN's
// (once an operator); a Newton step's, rebuilt at every step, are not (some 50 us less a
// step at 1025 x 513: a field of seven steps 12.4 ms against 12.8).
void build_hierarchy(bt_poisson *p, const double *reaction) {
    cudaStream_t st = p->ctx->stream;
    Timed timed(p->ctx, "hierarchy");
    Level &L0 = p->levels[0];
    BT_LAUNCH(p->ctx, add_diag, blocks_for(p->n, 256), 256, 0, st, p->n, L0.base.as<double>(p->n), reaction,
                                                    L0.active.as<uint8_t>(p->n),
                                                    L0.diag.as<double>(p->n), L0.rdiag.as<double>(p->n));
    if (reaction)
        coarse_operators<false>(p);
    else
        coarse_operators<true>(p);
    Level &Lc = p->levels.back();
    if (p->levels.size() == 1)
        BT_LAUNCH(p->ctx, five_to_nine, blocks_for(Lc.n, 256), 256, 0, st, Lc.n,
                  Lc.c4.as<double>(4 * Lc.n), Lc.diag.as<double>(Lc.n), Lc.active.as<uint8_t>(Lc.n),
                  Lc.a9.as<double>(9 * Lc.n));
    int *status = p->status.as<int>(2);  // [0] singular, [1] the banded path fell back
    BT_CUDA(cudaMemsetAsync(status, 0, 2 * sizeof(int), st));
    double *inv = p->inv.as<double>(Lc.n * Lc.n);
    const double *a9c = Lc.a9.as<double>(9 * Lc.n);
    if (band_half(Lc.nx, Lc.ny) <= kBandMax) {
        if (reaction)
            coarsest_band<false>(p, a9c, inv, status);
        else
            coarsest_band<true>(p, a9c, inv, status);
        BT_LAUNCH(p->ctx, coarsest_invert, 1, kInvertThreads, 0, st, Lc.nx, Lc.ny, a9c, inv,
                  status, status + 1);
    } else {
        BT_LAUNCH(p->ctx, coarsest_invert, 1, kInvertThreads, 0, st, Lc.nx, Lc.ny, a9c, inv,
                  status, (const int *)nullptr);
    }
    BT_CHECK_LAUNCH();
    refresh_tail_image(p);
    p->built = true;
    p->reaction_on = reaction != nullptr;
}

// The shared memory any solver's coarsest level needs.
template <bool PLAIN>
void coarsest_band_limits() {
    BT_CUDA(cudaFuncSetAttribute(coarsest_band_factor<PLAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * kCoarsest * (2 * kBandMax + 2))));
    const int solve = (int)(sizeof(double) * kCoarsest * (2 * kBandPad + 1));
    BT_CUDA(cudaFuncSetAttribute((coarsest_band_solve<6, PLAIN>), cudaFuncAttributeMaxDynamicSharedMemorySize, solve));
    BT_CUDA(cudaFuncSetAttribute((coarsest_band_solve<10, PLAIN>), cudaFuncAttributeMaxDynamicSharedMemorySize, solve));
    BT_CUDA(cudaFuncSetAttribute((coarsest_band_solve<14, PLAIN>), cudaFuncAttributeMaxDynamicSharedMemorySize, solve));
    BT_CUDA(cudaFuncSetAttribute((coarsest_band_solve<18, PLAIN>), cudaFuncAttributeMaxDynamicSharedMemorySize, solve));
}

// The tail: the longest run of coarsest levels (never level 0, whose operator is 5-point),
// each at most tail_nodes large, whose shared-memory image fits one block; its descriptors
// and layout, and the shared memory of the staged smoother.
void setup_tail(bt_poisson *p) {
    const int levels = (int)p->levels.size();
    p->tail_start = -1;
    p->tail_smem = 0;
    for (int l = levels - 1; l >= 1 && levels - l <= kTailMaxLevels; --l) {
        const Level &L = p->levels[l];
        if (L.n > p->tail_nodes || !tail_fits_threads(L.nx, L.ny) ||
            tail_layout(p->levels, l).total() > kTailSmemMax)
            break;
        p->tail_start = l;
    }
    // the largest band any solver's coarsest level needs (the attribute is the kernel's,
    // shared by every solver of the process: never set it to one mesh's own size)
    coarsest_band_limits<true>();
    coarsest_band_limits<false>();
    if (p->tail_start <= 0) return;
    const TailLayout T = tail_layout(p->levels, p->tail_start);
    p->tail_smem = T.total();
    p->tail_doubles = T.doubles;
    p->tail_ints = T.ints;
    p->tail_words = (int)(T.image() / 16);
    std::vector<TailLevel> tail;
    for (int l = p->tail_start; l < levels; ++l) {
        Level &L = p->levels[l];
        TailLevel t{};
        t.nx = L.nx;
        t.ny = L.ny;
        t.n = L.n;
        t.a9 = L.a9.as<double>(9 * L.n);
        t.rdiag = L.rdiag.as<double>(L.n);
        t.active = L.active.as<uint8_t>(L.n);
        t.x = L.x.as<double>(L.n);
        t.b = L.b.as<double>(L.n);
        tail.push_back(t);
    }
    // the largest any solver asks for: solvers of other meshes may launch concurrently
    BT_CUDA(cudaFuncSetAttribute(vcycle_tail, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kTailSmemMax));
    BT_CUDA(cudaMemcpy(p->tail_levels.as<TailLevel>(tail.size()), tail.data(),
                       sizeof(TailLevel) * tail.size(), cudaMemcpyHostToDevice));
    BT_CUDA(cudaMemcpy(p->tail_plans.as<TailPlan>(T.plan.size()), T.plan.data(),
                       sizeof(TailPlan) * T.plan.size(), cudaMemcpyHostToDevice));
    p->tail_image.get(T.image());
    refresh_tail_image(p, true);
}

// Copy the tail levels' coefficients and active flags into the tail's static image (after
// the hierarchy's coefficients change), with the transfer tables when it is laid out.
void refresh_tail_image(bt_poisson *p, bool tables) {
    if (p->tail_start <= 0) return;
    cudaStream_t st = p->ctx->stream;
    const TailLayout T = tail_layout(p->levels, p->tail_start);
    char *image = static_cast<char *>(p->tail_image.get(T.image()));
    double *d = reinterpret_cast<double *>(image);
    int32_t *ints = reinterpret_cast<int32_t *>(d + T.doubles);
    uint8_t *bytes = reinterpret_cast<uint8_t *>(ints + T.ints);
    auto copy = [&](void *dst, const void *src, size_t n) {
        if (n) BT_CUDA(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToDevice, st));
    };
    const int levels = (int)p->levels.size();
    for (int l = p->tail_start; l < levels; ++l) {
        Level &L = p->levels[l];
        const TailPlan &P = T.plan[l - p->tail_start];
        copy(bytes + P.act, L.active.as<uint8_t>(L.n), L.n);
        if (l + 1 == levels) continue;
        const Fine F = fine_of(L, p->levels[l + 1], false);
        copy(d + P.a9, L.a9.as<double>(9 * L.n), sizeof(double) * 9 * L.n);
        copy(d + P.rd, L.rdiag.as<double>(L.n), sizeof(double) * L.n);
        if (!tables) continue;
        copy(d + P.wx, F.wx, sizeof(double) * P.nx);
        copy(d + P.wy, F.wy, sizeof(double) * P.ny);
        copy(d + P.rxw, F.rxw, sizeof(double) * kRestrict * P.ncx);
        copy(d + P.ryw, F.ryw, sizeof(double) * kRestrict * P.ncy);
        copy(ints + P.lox, F.lox, sizeof(int32_t) * P.nx);
        copy(ints + P.loy, F.loy, sizeof(int32_t) * P.ny);
        copy(ints + P.rx0, F.rx0, sizeof(int32_t) * P.ncx);
        copy(ints + P.ry0, F.ry0, sizeof(int32_t) * P.ncy);
    }
}

void drop_graphs(bt_poisson *p) {
    if (p->vexec) cudaGraphExecDestroy(p->vexec);
    if (p->vgraph) cudaGraphDestroy(p->vgraph);
    p->vexec = nullptr;
    p->vgraph = nullptr;
}

// The smoothing of level l before (pre) or after the coarse correction: red-black sweeps
// on level 0, four-colour sweeps on 9-point levels, the colours reversed afterwards; the
// phases in shared-memory staged launches (up to kMaxPhases each) that move x between the
// level's two buffers, or one in-place launch per colour.
// The level's smoothing sweeps; with xc, after adding the prolonged coarse correction
// (P of the fine-coarse pair `pf`) to x: in the first staged launch's read of x, or by
// prolong_add.
void smooth(bt_poisson *p, size_t l, bool pre, const Fine *pf = nullptr,
            const double *xc = nullptr) {
    cudaStream_t st = p->ctx->stream;
    Level &L = p->levels[l];
    const int T = 256;
    const double *b = L.b.as<double>(L.n);
    const uint8_t *act = L.active.as<uint8_t>(L.n);
    const bool five = l == 0;
    const int colours = five ? 2 : 4;
    const int sweeps = five ? p->fine_sweeps : p->coarse_sweeps;
    if (p->staged) {
        const int tx = five ? kStage5X : kStage9X, ty = five ? kStage5Y : kStage9Y;
        const dim3 tiles((unsigned)((L.nx + tx - 1) / tx), (unsigned)((L.ny + ty - 1) / ty));
        const int phases = sweeps * colours;
        for (int start = 0; start < phases; start += kMaxPhases) {
            const int count = std::min(kMaxPhases, phases - start);
            double *x = L.x.as<double>(L.n);
            double *out = L.cur == x ? L.x2.as<double>(L.n) : x;
            SmoothView V{};
            V.nx = (int)L.nx;
            V.ny = (int)L.ny;
            V.n = L.n;
            V.c4 = five ? L.c4.as<double>(4 * L.n) : nullptr;
            V.a9 = five ? nullptr : L.a9.as<double>(9 * L.n);
            V.rdiag = L.rdiag.as<double>(L.n);
            V.b = b;
            V.active = act;
            V.xin = L.cur;
            V.xout = out;
            if (start == 0 && xc) {
                V.xc = xc;
                V.ax = CoarseAxis{(int)L.nx, (int)pf->ncx};
                V.ay = CoarseAxis{(int)L.ny, (int)pf->ncy};
            }
            const CycleIo *io = five ? p->cycle_io.as<CycleIo>(1) : nullptr;
            const bool first = pre && start == 0;  // every level's cycle starts from zero
            const bool last = five && !pre && start + count == phases;
#define BT_SMOOTH(N, X, Y, C)                                                                   \
    if (five != N && count == C) {                                                                \
        if (pre)                                                                                   \
            BT_LAUNCH(p->ctx, (smooth_level<N, X, Y, C, false>), tiles, (Tile<N, X, Y, C>::threads), \
                      0, st, V, io, first, last);                                                  \
        else                                                                                       \
            BT_LAUNCH(p->ctx, (smooth_level<N, X, Y, C, true>), tiles, (Tile<N, X, Y, C>::threads),  \
                      0, st, V, io, first, last);                                                  \
    }
            BT_SMOOTH(false, kStage5X, kStage5Y, 2)
            BT_SMOOTH(false, kStage5X, kStage5Y, 4)
            BT_SMOOTH(false, kStage5X, kStage5Y, 6)
            BT_SMOOTH(false, kStage5X, kStage5Y, 8)
            BT_SMOOTH(true, kStage9X, kStage9Y, 4)
            BT_SMOOTH(true, kStage9X, kStage9Y, 8)
#undef BT_SMOOTH
            L.cur = out;
        }
        return;
    }
    std::vector<int> order;
    for (int sw = 0; sw < sweeps; ++sw)
        for (int c = 0; c < colours; ++c) order.push_back(pre ? c : colours - 1 - c);
    double *x = L.cur;
    if (xc) BT_LAUNCH(p->ctx, prolong_add, blocks_for(L.n, T), T, 0, st, *pf, xc, x);
    for (int c : order) {
        if (five) {
            const i64 per = L.nx * ((L.ny + 1) / 2);
            BT_LAUNCH(p->ctx, smooth5, blocks_for(per, T), T, 0, st, L.nx, L.ny,
                      L.c4.as<double>(4 * L.n), L.rdiag.as<double>(L.n), act, b, x, c);
        } else {
            const i64 per = colour_count(L.nx, L.ny, c);
            BT_LAUNCH(p->ctx, smooth9, blocks_for(per, T), T, 0, st, L.nx, L.ny,
                      L.a9.as<double>(9 * L.n), L.rdiag.as<double>(L.n), act, b, x, c);
        }
    }
}

// x = V-cycle(b) on level l (x starts at zero on entry for l > 0; level 0 takes b from, and
// leaves x in, the vectors the solver's CycleIo names).  The staged smoother moves a level's
// x between its two buffers; the cycle leaves it in the first.
void vcycle(bt_poisson *p, size_t l) {
    cudaStream_t st = p->ctx->stream;
    Level &L = p->levels[l];
    const int T = 256;
    if ((int)l == p->tail_start) {
        const int count = (int)(p->levels.size() - l);
        const Level &Lc = p->levels.back();
        BT_LAUNCH(p->ctx, vcycle_tail, kTailCluster, kTailThreads, p->tail_smem, st,
                  p->tail_levels.as<TailLevel>(count), p->tail_plans.as<TailPlan>(count), count,
                  static_cast<const uint4 *>(p->tail_image.get(16 * (size_t)p->tail_words)),
                  p->tail_words, p->tail_doubles, p->tail_ints, p->inv.as<double>(Lc.n * Lc.n),
                  p->coarse_sweeps);
        return;
    }
    if (l + 1 == p->levels.size()) {
        BT_LAUNCH(p->ctx, coarsest_apply, 1, kCoarsest, 0, st, (int)L.n, p->inv.as<double>(L.n * L.n),
                  L.active.as<uint8_t>(L.n), L.b.as<double>(L.n), L.x.as<double>(L.n),
                  l == 0 ? p->cycle_io.as<CycleIo>(1) : nullptr);
        return;
    }
    Level &C = p->levels[l + 1];
    double *b = L.b.as<double>(L.n);
    const uint8_t *act = L.active.as<uint8_t>(L.n);
    L.cur = L.x.as<double>(L.n);
    const CycleIo *io = l == 0 ? p->cycle_io.as<CycleIo>(1) : nullptr;
    if (io && !p->staged)
        BT_LAUNCH(p->ctx, cycle_begin, blocks_for(L.n, T), T, 0, st, io, L.n, b, L.cur);
    smooth(p, l, true);
    Fine F = fine_of(L, C, l == 0);
    RestrictView R{};
    R.nx = (int)L.nx;
    R.ny = (int)L.ny;
    R.ncx = (int)C.nx;
    R.ncy = (int)C.ny;
    R.n = L.n;
    R.c4 = F.c4;
    R.diag = F.diag;
    R.a9 = F.a9;
    R.weight = F.weight;
    R.active = act;
    R.x = L.cur;
    R.b = b;
    R.bc = C.b.as<double>(C.n);
    const dim3 tiles((unsigned)((C.nx + kRestrictX - 1) / kRestrictX),
                     (unsigned)((C.ny + kRestrictY - 1) / kRestrictY));
    if (l == 0)
        BT_LAUNCH(p->ctx, restrict_level<false>, tiles, kRestrictThreads, 0, st, R, io);
    else
        BT_LAUNCH(p->ctx, restrict_level<true>, tiles, kRestrictThreads, 0, st, R, io);
    if (!p->staged)  // (the staged smoothing starts from zero by itself)
        BT_LAUNCH(p->ctx, fill_zero, blocks_for(C.n, T), T, 0, st, C.n, C.x.as<double>(C.n));
    vcycle(p, l + 1);
    smooth(p, l, false, &F, C.x.as<double>(C.n));
    if (io) {
        if (!p->staged) BT_LAUNCH(p->ctx, cycle_end, blocks_for(L.n, T), T, 0, st, io, L.n, L.cur);
        BT_CHECK_LAUNCH();
        return;
    }
    if (L.cur != L.x.as<double>(L.n))
        BT_CUDA(cudaMemcpyAsync(L.x.as<double>(L.n), L.cur, sizeof(double) * L.n,
                                cudaMemcpyDeviceToDevice, st));
    L.cur = L.x.as<double>(L.n);
    BT_CHECK_LAUNCH();
}

// Capture the V-cycle (from the vector CycleIo::b to CycleIo::z) as a graph: every other
// buffer it touches keeps its address for the solver's life, so one capture serves every
// solve and every Newton Jacobian (whose coefficients change in place).
void capture_vcycle(bt_poisson *p) {
    // captured on the context's own stream (the default stream cannot capture); the
    // graph then runs on whichever stream the context queues on
    cudaStream_t st = p->ctx->own_stream;
    cudaStream_t queue = p->ctx->stream;
    p->cycle_io.as<CycleIo>(1);  // (allocated before the capture)
    const i64 before = p->ctx->launch_count;
    p->ctx->stream = st;
    BT_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    try {
        vcycle(p, 0);
    } catch (...) {
        cudaGraph_t broken = nullptr;
        cudaStreamEndCapture(st, &broken);
        if (broken) cudaGraphDestroy(broken);
        p->ctx->stream = queue;
        throw;
    }
    p->ctx->stream = queue;
    BT_CUDA(cudaStreamEndCapture(st, &p->vgraph));
    BT_CUDA(cudaGraphInstantiate(&p->vexec, p->vgraph, 0));
    p->vgraph_kernels = p->ctx->launch_count - before;
    p->ctx->launch_count = before;  // counted when the graph runs
}

// One V-cycle from zero, from CycleIo::b to CycleIo::z.
void run_cycle(bt_poisson *p) {
    if (!p->vexec) capture_vcycle(p);
    {
        Timed timed(p->ctx, "vcycle");
        BT_CUDA(cudaGraphLaunch(p->vexec, p->ctx->stream));
    }
    p->ctx->launch_count += p->vgraph_kernels;
}

// z = M v: one V-cycle from zero.  Blocks of the cycle's last launch read v around the nodes
// of z that others write: where the two overlap, v's copy in the level's own b is read instead.
void precondition(bt_poisson *p, const double *v, double *z) {
    if (v < z + p->n && z < v + p->n) {
        double *b = p->levels[0].b.as<double>(p->n);
        BT_CUDA(cudaMemcpyAsync(b, v, sizeof(double) * p->n, cudaMemcpyDeviceToDevice, p->ctx->stream));
        v = b;
    }
    BT_LAUNCH(p->ctx, set_cycle, 1, 1, 0, p->ctx->stream, p->cycle_io.as<CycleIo>(1), v, z);
    run_cycle(p);
}

// `count` device doubles, read after the queued work.
const double *read_scalars(bt_poisson *p, const double *dev, int count) {
    double *host = static_cast<double *>(p->ctx->host.get(sizeof(double) * 64));
    BT_CUDA(cudaMemcpyAsync(host, dev, sizeof(double) * count, cudaMemcpyDeviceToHost, p->ctx->stream));
    BT_CUDA(cudaStreamSynchronize(p->ctx->stream));
    return host;
}

// The finishing-block counter of the passes over vectors (zero between them) and the blocks'
// partial sums.
unsigned *dot_ticket(bt_poisson *p) {
    unsigned *ticket = p->dot_ticket.as<unsigned>(1);
    if (!p->ticket_ready) {
        BT_CUDA(cudaMemsetAsync(ticket, 0, sizeof(unsigned), p->ctx->stream));
        p->ticket_ready = true;
    }
    return ticket;
}
double *dot_partial(bt_poisson *p) {
    return p->dot_partial.as<double>((size_t)kDotBlocks * kDotMax);
}

Rows5 rows_of(bt_poisson *p) {
    Level &L = p->levels[0];
    return Rows5{L.nx, L.ny, L.c4.as<double>(4 * L.n), L.diag.as<double>(L.n),
                 L.active.as<uint8_t>(L.n)};
}

// One pass of Krylov step S.j.
template <int MODE>
void krylov_launch(bt_poisson *p, const ArnoldiState &S, const double *V, const double *z, double *w) {
    const int m = S.j + 1;
    cudaStream_t st = p->ctx->stream;
    double *partial = dot_partial(p);
    unsigned *ticket = dot_ticket(p);
    const Rows5 A = rows_of(p);
    BT_REQUIRE(m >= 1 && m <= kDotMax, "poisson: a Krylov pass takes 1 to 32 vectors");
#define BT_PASS(MQ)                                                                             \
    BT_LAUNCH(p->ctx, (krylov_pass<MQ, MODE>), dot_blocks(p->n), kDotThreads, 0, st, A, V, z, w,  \
              p->n, m, S, partial, ticket)
    if (m <= 4)
        BT_PASS(4);
    else if (m <= 8)
        BT_PASS(8);
    else if (m <= 16)
        BT_PASS(16);
    else
        BT_PASS(32);
#undef BT_PASS
}

// r = u - A x and the norms of u and r (one launch and one read)
struct Norms {
    double u, r;
};
Norms residual(bt_poisson *p, const double *u, const double *x, double *r) {
    double *s = p->scalars.as<double>(16);
    BT_LAUNCH(p->ctx, residual_norms, dot_blocks(p->n), kDotThreads, 0, p->ctx->stream, rows_of(p), u,
              x, p->n, r, dot_partial(p), dot_ticket(p), s);
    BT_CHECK_LAUNCH();
    const double *host = read_scalars(p, s, 2);
    return {std::sqrt(host[0]), std::sqrt(host[1])};
}

double norm2(bt_poisson *p, const double *v) {
    double *s = p->scalars.as<double>(16);
    BT_LAUNCH(p->ctx, vector_norm, dot_blocks(p->n), kDotThreads, 0, p->ctx->stream, v, p->n,
              dot_partial(p), dot_ticket(p), s);
    BT_CHECK_LAUNCH();
    return std::sqrt(read_scalars(p, s, 1)[0]);
}

// The steps a cycle still needs by the rate of its last (up to three) steps, one fewer so
// that a queued step rarely runs past the end: at least 1.
int steps_to_queue(const Arnoldi &a) {
    const int j = a.j;
    const int k = std::min(j, 3);
    const double r = a.resid[j];
    if (k == 0 || !(r > 0.0) || !(a.resid[j - k] > 0.0)) return 1;
    const double rate = std::pow(r / a.resid[j - k], 1.0 / k);
    if (!(rate < 0.95)) return 1;
    const double left = std::log(a.tol / r) / std::log(rate);
    if (!(left < 1e6)) return 1;
    return std::max(1, (int)std::ceil(left) - 1);
}

// A residual norm, which must be finite: no comparison with a tolerance would tell that it is
// not (one that is no number fails them all, and a tolerance relative to an infinite one is met).
double finite_norm(double norm) {
    if (!std::isfinite(norm)) throw Error{BT_ERR_NOCONV, "field solve: the residual is not finite"};
    return norm;
}

// Solve A d = r0 for d (d zero on entry, beta = |r0|) by restarted right-preconditioned GMRES
// until ||r0 - A d|| <= abs_tol or max_iter V-cycles; returns the V-cycles run and the final
// residual norm.  The Arnoldi process runs on the device (Gram-Schmidt twice, the Givens
// rotations in arnoldi_step); the host queues steps in batches sized by the residual's
// rate and reads the state between them, and the cycle's solution is the same as if it
// read it after every step.
int gmres(bt_poisson *p, const double *r0, double *d, double beta, double abs_tol, int max_iter,
          double *final_norm) {
    const i64 n = p->n;
    const int m = p->restart;  // at most kDotMax - 1: a basis of m + 1 vectors
    cudaStream_t st = p->ctx->stream;
    double *V = p->V.as<double>((size_t)(m + 1) * n);
    double *Z = p->Z.as<double>((size_t)(m + 1) * n);
    double *w = p->work.as<double>(n);
    CycleIo *io = p->cycle_io.as<CycleIo>(1);
    // the device state: Arnoldi, H, cs, sn, g, y and the passes' coefficients and norm
    const size_t head = (sizeof(Arnoldi) + 255) / 256 * 256;
    const size_t doubles = (size_t)(m + 1) * m + 3 * m + 1 + 2 * (m + 2) + 1;
    unsigned char *state = p->arnoldi.as<unsigned char>(head + sizeof(double) * doubles);
    ArnoldiState S{};
    S.a = reinterpret_cast<Arnoldi *>(state);
    S.H = reinterpret_cast<double *>(state + head);
    S.cs = S.H + (size_t)(m + 1) * m;
    S.sn = S.cs + m;
    S.g = S.sn + m;
    double *y = S.g + m + 1;
    S.h1 = y + m;
    S.h2 = S.h1 + (m + 2);
    S.hn = S.h2 + (m + 2);
    S.m = m;
    Arnoldi *host = static_cast<Arnoldi *>(p->ctx->host.get(std::max(sizeof(Arnoldi), 64 * sizeof(double))));
    int total = 0;
    const double *r = r0;
    finite_norm(beta);
    double previous = INFINITY;
    // stop at the tolerance, or where a whole restart cycle no longer halves the true
    // residual: the rounding floor of the residual itself
    while (beta > abs_tol && total < max_iter && beta < 0.5 * previous) {
        previous = beta;
        BT_LAUNCH(p->ctx, arnoldi_begin, blocks_for(n, 256), 256, 0, st, S.a, S.g, m, beta, abs_tol, r,
                  n, V, Z, io);
        int j = 0, batch = 2;
        for (;;) {
            const int count = std::min(batch, std::min(m - j, max_iter - total));
            for (int b = 0; b < count; ++b, ++j, ++total) {
                S.j = j;
                const double *z = Z + (i64)j * n;
                run_cycle(p);
                krylov_launch<kApply>(p, S, V, z, w);
                krylov_launch<kOrthDots>(p, S, V, z, w);
                krylov_launch<kOrthNorm>(p, S, V, z, w);
                BT_LAUNCH(p->ctx, scale_by_norm, blocks_for(n, 256), 256, 0, st, w, S.hn, n,
                          V + (i64)(j + 1) * n, Z + (i64)(j + 1) * n, io);
            }
            BT_CHECK_LAUNCH();
            BT_CUDA(cudaMemcpyAsync(host, S.a, sizeof(Arnoldi), cudaMemcpyDeviceToHost, st));
            BT_CUDA(cudaStreamSynchronize(st));
            if (host->done || j >= m || total >= max_iter) break;
            batch = steps_to_queue(*host);
        }
        // d += Z y, y = H^-1 g over the steps taken
        BT_LAUNCH(p->ctx, arnoldi_solve, 1, 32, 0, st, S.a, S.H, S.g, y, m);
        BT_LAUNCH(p->ctx, combine, blocks_for(n, 256), 256, 0, st, Z, y, S.a, n, d);
        // the true residual r0 - A d
        beta = finite_norm(residual(p, r0, d, w).r);
        r = w;
    }
    if (final_norm) *final_norm = beta;
    return total;
}

}  // namespace
}  // namespace bt

extern "C" int bt_poisson_create(bt_ctx *ctx, const bt_mesh_desc *m, bt_poisson **out) {
    return bt::guarded([&] {
        BT_REQUIRE(ctx && m && out, "poisson: null argument");
        BT_REQUIRE(m->nx >= 3 && m->ny >= 3, "poisson: the mesh needs at least 3 nodes per axis");
        BT_REQUIRE(m->x && m->fixed && m->fixed_value && m->distance, "poisson: null mesh array");
        BT_REQUIRE(m->h > 0.0, "poisson: h must be positive");
        auto p = new bt_poisson;
        try {
            p->ctx = ctx;
            p->nx = m->nx;
            p->ny = m->ny;
            p->n = m->nx * m->ny;
            p->h = m->h;
            p->cyl = m->cylindrical;
            if (p->cyl) {
                const double rows = m->origin_y / m->h;
                p->j0 = (i64)llround(rows);
                BT_REQUIRE(p->j0 >= 0 && std::fabs(rows - (double)p->j0) <= 1e-6,
                           "poisson: a cylindrical mesh starts on the axis or a multiple of h "
                           "above it");
            }
            for (int q = 0; q < 4; ++q) p->neumann[q] = m->neumann ? m->neumann[q] : 0.0;
            const i64 n = p->n;
            BT_CUDA(cudaMemcpy(p->x.as<double>(p->nx), m->x, sizeof(double) * p->nx, cudaMemcpyHostToDevice));
            BT_CUDA(cudaMemcpy(p->fixed.as<uint8_t>(n), m->fixed, n, cudaMemcpyHostToDevice));
            BT_CUDA(cudaMemcpy(p->value.as<double>(n), m->fixed_value, sizeof(double) * n, cudaMemcpyHostToDevice));
            BT_CUDA(cudaMemcpy(p->distance.as<double>(4 * n), m->distance, sizeof(double) * 4 * n, cudaMemcpyHostToDevice));
            BT_CUDA(cudaMemcpy(p->fixed_eff.as<uint8_t>(n), m->fixed, n, cudaMemcpyHostToDevice));
            BT_CUDA(cudaMemcpy(p->value_eff.as<double>(n), m->fixed_value, sizeof(double) * n, cudaMemcpyHostToDevice));
            // the levels
            p->levels.reserve(48);
            i64 nx = p->nx, ny = p->ny;
            while (true) {
                p->levels.emplace_back();
                bt::Level &L = p->levels.back();
                L.nx = nx;
                L.ny = ny;
                L.n = nx * ny;
                L.x.as<double>(L.n);
                L.x2.as<double>(L.n);
                L.b.as<double>(L.n);
                L.active.as<uint8_t>(L.n);
                L.rdiag.as<double>(L.n);
                if (p->levels.size() == 1) {
                    L.c4.as<double>(4 * L.n);
                    L.diag.as<double>(L.n);
                    L.base.as<double>(L.n);
                    L.weight.as<double>(L.n);
                } else {
                    L.a9.as<double>(9 * L.n);
                }
                const bool more = L.n > bt::kCoarsest && (nx > 3 || ny > 3);
                if (!more) break;
                bt::build_axis(L.ax, nx);
                bt::build_axis(L.ay, ny);
                nx = L.ax.nc;
                ny = L.ay.nc;
            }
            BT_REQUIRE(p->levels.back().n <= bt::kCoarsest, "poisson: coarsest level too large");
            bt::setup_tail(p);
            p->src.as<double>(n);
            bt::build_operator(p);
            BT_CUDA(cudaStreamSynchronize(ctx->stream));
        } catch (...) {
            delete p;
            throw;
        }
        *out = p;
    });
}

extern "C" int bt_poisson_destroy(bt_poisson *p) {
    return bt::guarded([&] {
        if (!p) return;
        cudaStreamSynchronize(p->ctx->stream);
        delete p;
    });
}

extern "C" int bt_poisson_set_region(bt_poisson *p, const uint8_t *mask, double value) {
    return bt::guarded([&] {
        BT_REQUIRE(p, "poisson: null solver");
        const i64 n = p->n;
        std::vector<uint8_t> fixed(n);
        std::vector<double> val(n);
        BT_CUDA(cudaMemcpy(fixed.data(), p->fixed.as<uint8_t>(n), n, cudaMemcpyDeviceToHost));
        BT_CUDA(cudaMemcpy(val.data(), p->value.as<double>(n), sizeof(double) * n, cudaMemcpyDeviceToHost));
        if (mask)
            for (i64 f = 0; f < n; ++f)
                if (mask[f] && !fixed[f]) {
                    fixed[f] = 1;
                    val[f] = value;
                }
        BT_CUDA(cudaMemcpy(p->fixed_eff.as<uint8_t>(n), fixed.data(), n, cudaMemcpyHostToDevice));
        BT_CUDA(cudaMemcpy(p->value_eff.as<double>(n), val.data(), sizeof(double) * n, cudaMemcpyHostToDevice));
        p->has_region = mask != nullptr;
        p->region_value = value;
        bt::build_operator(p);
    });
}

extern "C" int bt_poisson_solve(bt_poisson *p, double *phi, const double *rho, double amplitude,
                                double temperature, double up, int32_t sign, double tol,
                                double newton_tol, int32_t max_newton, int32_t *newton_steps,
                                int32_t *cycles) {
    return bt::guarded([&] {
        BT_REQUIRE(p && phi, "poisson: null argument");
        BT_REQUIRE(tol > 0.0, "poisson: the tolerance must be positive");
        const i64 n = p->n;
        cudaStream_t st = p->ctx->stream;
        bt::Level &L0 = p->levels[0];
        double *b = p->rhs.as<double>(n);
        double *r0 = p->r0.as<double>(n);
        double *d = p->delta.as<double>(n);
        double *reaction = p->reaction.as<double>(n);
        double *scal = p->scalars.as<double>(16);
        const int max_cycles = 4000;
        bt::Timed timed(p->ctx, "field_solve");
        BT_LAUNCH(p->ctx, bt::prepare, bt::blocks_for(n, 256), 256, 0, st, n, rho, p->src.as<double>(n), L0.active.as<uint8_t>(n), p->value_eff.as<double>(n),
            b, phi);
        BT_CHECK_LAUNCH();
        int total_cycles = 0, steps = 0;
        BT_REQUIRE(!p->transposed || !(amplitude > 0.0),
                   "poisson: the transposed solver takes linear solves only");
        const double *weight = L0.weight.as<double>(n);
        const uint8_t *active = L0.active.as<uint8_t>(n);
        if (p->transposed) {  // A^T z = b as B y = W^-1 b, y = W^-1 z (transpose_c4)
            BT_LAUNCH(p->ctx, bt::scale_by_weight, bt::blocks_for(n, 256), 256, 0, st, n, weight, active, 1, b);
            BT_LAUNCH(p->ctx, bt::scale_by_weight, bt::blocks_for(n, 256), 256, 0, st, n, weight, active, 1, phi);
        }
        if (!(amplitude > 0.0)) {
            if (!p->built || p->reaction_on) bt::build_hierarchy(p, nullptr);
            // r0 = b - A phi; the tolerance is relative to the larger of |b| and |r0|
            const bt::Norms norms = bt::residual(p, b, phi, r0);
            const double scale = std::max(norms.u, norms.r);
            BT_CUDA(cudaMemsetAsync(d, 0, sizeof(double) * n, st));
            double left = 0.0;
            const double goal = tol * (scale > 0.0 ? scale : 1.0);
            total_cycles = bt::gmres(p, r0, d, norms.r, goal, max_cycles, &left);
            BT_LAUNCH(p->ctx, bt::add_into, bt::blocks_for(n, 256), 256, 0, st, d, n, phi);
            if (p->transposed)
                BT_LAUNCH(p->ctx, bt::scale_by_weight, bt::blocks_for(n, 256), 256, 0, st, n, weight, active, 0, phi);
            BT_CHECK_LAUNCH();
            // a residual stalled within 1e4 of the goal is the floor of its own rounding
            if (!(left <= 1e4 * goal))
                throw bt::Error{BT_ERR_NOCONV, "field solve: GMRES did not reach the tolerance"};
        } else {
            BT_REQUIRE(temperature > 0.0, "poisson: the temperature must be positive");
            BT_REQUIRE(sign == 1 || sign == -1, "poisson: the species' sign must be +-1");
            const int limit = max_newton > 0 ? max_newton : 100;
            bool converged = false;
            for (steps = 1; steps <= limit; ++steps) {
                BT_LAUNCH(p->ctx, bt::boltzmann, bt::blocks_for(n, 256), 256, 0, st, p->nx, p->ny, L0.c4.as<double>(4 * n), L0.base.as<double>(n),
                    L0.active.as<uint8_t>(n), phi, b, amplitude, temperature, up, (double)sign,
                    r0, reaction);
                BT_CHECK_LAUNCH();
                bt::build_hierarchy(p, reaction);
                const double fnorm = bt::norm2(p, r0);
                BT_CUDA(cudaMemsetAsync(d, 0, sizeof(double) * n, st));
                double left = 0.0;
                total_cycles += bt::gmres(p, r0, d, fnorm, tol * (fnorm > 0.0 ? fnorm : 1.0),
                                          max_cycles, &left);
                BT_LAUNCH(p->ctx, bt::add_max, bt::dot_blocks(n), bt::kDotThreads, 0, st, d, n, phi,
                          bt::dot_partial(p), bt::dot_ticket(p), scal + 8);
                BT_CHECK_LAUNCH();
                const double change = bt::read_scalars(p, scal + 8, 1)[0];
                if (!std::isfinite(change))
                    throw bt::Error{BT_ERR_NOCONV, "field solve: Newton's update is not finite"};
                if (change < newton_tol) {
                    converged = true;
                    break;
                }
            }
            if (!converged) steps = limit;
        }
        int status = 0;
        BT_CUDA(cudaMemcpyAsync(&status, p->status.as<int>(1), sizeof(int), cudaMemcpyDeviceToHost, st));
        BT_CUDA(cudaStreamSynchronize(st));
        if (status)
            throw bt::Error{BT_ERR_NOCONV, "field solve: the coarsest operator is singular (is any node held?)"};
        if (newton_steps) *newton_steps = steps;
        if (cycles) *cycles = total_cycles;
    });
}

namespace bt {
namespace {
// r = rho / eps0 + c - A phi on the free nodes of the level-0 operator (its diagonal
// without a Newton reaction), 0 on the held ones
__global__ void linear_residual(i64 nx, i64 ny, const double *__restrict__ c4,
                                const double *__restrict__ base, const double *__restrict__ src,
                                const uint8_t *__restrict__ active, const double *__restrict__ phi,
                                const double *__restrict__ rho, double *__restrict__ r) {
    const i64 n = nx * ny;
    const i64 f = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n) return;
    if (!active[f]) {
        r[f] = 0.0;
        return;
    }
    const i64 i = f / ny, j = f - i * ny;
    double s = base[f] * phi[f];
    if (i > 0) s -= c4[f] * phi[f - ny];
    if (i < nx - 1) s -= c4[n + f] * phi[f + ny];
    if (j > 0) s -= c4[2 * n + f] * phi[f - 1];
    if (j < ny - 1) s -= c4[3 * n + f] * phi[f + 1];
    r[f] = (rho ? rho[f] / kEps0 : 0.0) + src[f] - s;
}
}  // namespace
}  // namespace bt

extern "C" int bt_poisson_residual(bt_poisson *p, const double *phi, const double *rho,
                                   double *r) {
    return bt::guarded([&] {
        BT_REQUIRE(p && phi && r, "poisson residual: null argument");
        BT_REQUIRE(!p->transposed, "poisson residual: the solver is transposed");
        const i64 n = p->n;
        bt::Level &L0 = p->levels[0];
        BT_LAUNCH(p->ctx, bt::linear_residual, bt::blocks_for(n, 256), 256, 0, p->ctx->stream, p->nx, p->ny,
                  L0.c4.as<double>(4 * n), L0.base.as<double>(n), p->src.as<double>(n),
                  L0.active.as<uint8_t>(n), phi, rho, r);
        BT_CHECK_LAUNCH();
    });
}

extern "C" int bt_poisson_solve_reaction(bt_poisson *p, double *phi, const double *rho,
                                         const double *reaction, double tol, int32_t *cycles) {
    return bt::guarded([&] {
        BT_REQUIRE(p && phi && reaction, "poisson: null argument");
        BT_REQUIRE(tol > 0.0, "poisson: the tolerance must be positive");
        BT_REQUIRE(!p->transposed, "poisson: the transposed solver takes no reaction");
        const i64 n = p->n;
        cudaStream_t st = p->ctx->stream;
        bt::Level &L0 = p->levels[0];
        double *b = p->rhs.as<double>(n);
        double *r0 = p->r0.as<double>(n);
        double *d = p->delta.as<double>(n);
        bt::Timed timed(p->ctx, "field_solve");
        BT_LAUNCH(p->ctx, bt::prepare, bt::blocks_for(n, 256), 256, 0, st, n, rho, p->src.as<double>(n),
                  L0.active.as<uint8_t>(n), p->value_eff.as<double>(n), b, phi);
        bt::build_hierarchy(p, reaction);
        const bt::Norms norms = bt::residual(p, b, phi, r0);
        const double scale = std::max(norms.u, norms.r);
        BT_CUDA(cudaMemsetAsync(d, 0, sizeof(double) * n, st));
        double left = 0.0;
        const double goal = tol * (scale > 0.0 ? scale : 1.0);
        const int total = bt::gmres(p, r0, d, norms.r, goal, 4000, &left);
        BT_LAUNCH(p->ctx, bt::add_into, bt::blocks_for(n, 256), 256, 0, st, d, n, phi);
        BT_CHECK_LAUNCH();
        if (!(left <= 1e4 * goal))
            throw bt::Error{BT_ERR_NOCONV, "field solve: GMRES did not reach the tolerance"};
        int status = 0;
        BT_CUDA(cudaMemcpyAsync(&status, p->status.as<int>(1), sizeof(int), cudaMemcpyDeviceToHost, st));
        BT_CUDA(cudaStreamSynchronize(st));
        if (status)
            throw bt::Error{BT_ERR_NOCONV, "field solve: the coarsest operator is singular (is any node held?)"};
        if (cycles) *cycles = total;
    });
}

extern "C" int bt_poisson_vcycle(bt_poisson *p, const double *b, const double *reaction,
                                 int32_t rebuild, double *z) {
    return bt::guarded([&] {
        BT_REQUIRE(p && b && z, "poisson: null argument");
        BT_REQUIRE(!p->transposed, "poisson: the transposed solver takes no V-cycle here");
        if (rebuild || !p->built || p->reaction_on != (reaction != nullptr))
            bt::build_hierarchy(p, reaction);
        bt::precondition(p, b, z);
        BT_CHECK_LAUNCH();
    });
}

extern "C" int bt_poisson_set_transposed(bt_poisson *p, int32_t on) {
    return bt::guarded([&] {
        BT_REQUIRE(p, "poisson: null solver");
        if ((on != 0) == p->transposed) return;
        BT_CUDA(cudaStreamSynchronize(p->ctx->stream));
        p->transposed = on != 0;
        bt::build_operator(p);
    });
}

extern "C" int bt_poisson_fixed_adjoint(bt_poisson *p, const double *z, const double *phi_bar,
                                        double *out) {
    return bt::guarded([&] {
        BT_REQUIRE(p && z && phi_bar && out, "poisson: null argument");
        const i64 n = p->n;
        bt::Level &L0 = p->levels[0];
        const double *c4 = p->transposed ? p->c4_plain.as<double>(4 * n) : L0.c4.as<double>(4 * n);
        BT_LAUNCH(p->ctx, bt::fixed_adjoint, bt::blocks_for(n, 256), 256, 0, p->ctx->stream,
                  p->nx, p->ny, c4, L0.active.as<uint8_t>(n), z, phi_bar, out);
        BT_CHECK_LAUNCH();
    });
}

extern "C" int bt_poisson_set_options(bt_poisson *p, int32_t fine_sweeps, int32_t coarse_sweeps,
                                      int32_t staged, int64_t tail_nodes) {
    return bt::guarded([&] {
        BT_REQUIRE(p, "poisson: null solver");
        BT_REQUIRE(fine_sweeps >= 1 && fine_sweeps <= 4, "poisson: fine_sweeps must be 1 to 4");
        BT_REQUIRE(coarse_sweeps >= 1 && coarse_sweeps <= 4,
                   "poisson: coarse_sweeps must be 1 to 4");
        BT_REQUIRE(tail_nodes >= 1, "poisson: tail_nodes must be positive");
        BT_CUDA(cudaStreamSynchronize(p->ctx->stream));
        p->fine_sweeps = fine_sweeps;
        p->coarse_sweeps = coarse_sweeps;
        p->staged = staged != 0;
        p->tail_nodes = tail_nodes;
        bt::drop_graphs(p);
        bt::setup_tail(p);
    });
}

// -- the batched field solve --------------------------------------------------------------
//
// Many candidates' linear field solves at once: each candidate keeps its own solver (its
// operator and multigrid hierarchy, built as for a single solve), and one launch per level
// step covers the level of every candidate that has it -- a table of (candidate, level)
// entries and the first block of each, so a block finds its entry by bisection.  The
// candidates' hierarchies are aligned at their finest levels: step l holds level l of every
// candidate whose one-block tail starts below l; the tails of all candidates run in one
// launch of one block each.  The iteration is multigrid's own: d <- d + V(r0 - A d), each
// candidate until its residual meets the single solve's criterion (|r| <= tol max(|b|,
// |r0|)) or stops falling (its rounding floor); a candidate that has stopped leaves every
// launch (its live flag), so the tables stay fixed for the batch's life.

namespace bt {
namespace {

constexpr int kBatchThreads = 256;

// One (candidate, level) of a level step: the level's arrays and its transfer to the next.
struct BatchLevel {
    int cand;
    i64 nx, ny, n;
    const double *c4, *diag, *a9;  // level 0: c4, diag; coarse levels: a9
    const uint8_t *active;
    double *x, *x2, *b;
    Fine F;           // to the next level
    double *xc, *bc;  // the next level's x and b
};

// One candidate's finest level for the outer iteration.
struct BatchFine {
    int cand;
    i64 nx, ny, n;
    const double *c4, *diag, *src, *value;
    const uint8_t *active;
    double *phi;        // its part of the batch's potential
    const double *rho;  // and of the density
    double *b, *r0, *d;
    double *vb, *vx;    // level 0's b and x: the V-cycle's input and output
};

struct BatchTail {
    int cand;
    const TailLevel *levels;
    const TailPlan *plans;
    int count;
    const uint4 *image;
    int words, doubles, ints;
    const double *inv;
    int sweeps;
};

// The entry of block `block`: the last whose first block is at or before it.
__device__ __forceinline__ int find_entry(const int *__restrict__ start, int n, int block) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(start + mid) <= block)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// Smoothing phases of every entry's level, a staged tile a block: from one of the level's
// x buffers (0: x, 1: x2) into the other; `zero_in`: x starts at zero (not read);
// `prolong`: the prolonged coarse correction is added as x is read.
template <bool NINE, int R>
__global__ void __launch_bounds__(kStageThreads)
    batch_smooth(const BatchLevel *__restrict__ E, const int *__restrict__ ids,
                 const int *__restrict__ start, int ne, const uint8_t *__restrict__ live,
                 int tx, int ty, Phases ph, int from, int prolong, int zero_in) {
    const int slot = find_entry(start, ne, blockIdx.x);
    const BatchLevel &L = E[ids[slot]];
    if (!live[L.cand]) return;
    const i64 local = (i64)blockIdx.x - start[slot];
    const i64 tiles_y = (L.ny + ty - 1) / ty;
    const i64 bx = local / tiles_y, by = local - bx * tiles_y;
    const double *in = from ? L.x2 : L.x;
    double *out = from ? L.x : L.x2;
    const Fine none{};
    smooth_staged_tile<NINE, R>(L.nx, L.ny, L.c4, L.diag, L.a9, L.active, L.b, in, out, tx, ty,
                                ph, prolong ? L.F : none, prolong ? L.xc : nullptr, bx, by,
                                zero_in != 0);
}

// The same in the register form, for the tiles the compiler knows (smooth_tile).
template <bool NINE, int TX, int TY, int COUNT, bool REVERSE>
__global__ void __launch_bounds__(Tile<NINE, TX, TY, COUNT>::threads)
    batch_smooth_tile(const BatchLevel *__restrict__ E, const int *__restrict__ ids,
                      const int *__restrict__ start, int ne, const uint8_t *__restrict__ live,
                      int from, int prolong, int zero_in) {
    const int slot = find_entry(start, ne, blockIdx.x);
    const BatchLevel &L = E[ids[slot]];
    if (!live[L.cand]) return;
    const int local = (int)blockIdx.x - start[slot];
    const int tiles_y = ((int)L.ny + TY - 1) / TY;
    const int bx = local / tiles_y, by = local - bx * tiles_y;
    SmoothView V{};
    V.nx = (int)L.nx;
    V.ny = (int)L.ny;
    V.n = L.n;
    V.c4 = L.c4;
    V.a9 = L.a9;
    V.rdiag = NINE ? L.a9 + 4 * L.n : L.diag;
    V.b = L.b;
    V.active = L.active;
    V.xin = zero_in ? nullptr : (from ? L.x2 : L.x);
    V.xout = from ? L.x : L.x2;
    V.xc = prolong ? L.xc : nullptr;
    V.ax = CoarseAxis{V.nx, (int)L.F.ncx};
    V.ay = CoarseAxis{V.ny, (int)L.F.ncy};
    smooth_tile<NINE, TX, TY, COUNT, REVERSE, true>(V, bx, by);
}

// b of the next level = R (b - A x) on every entry's level (x in the buffer `from` names:
// 0 x, 1 x2).
template <bool NINE>
__global__ void __launch_bounds__(kRestrictThreads)
    batch_restrict(const BatchLevel *__restrict__ E, const int *__restrict__ ids,
                   const int *__restrict__ start, int ne, const uint8_t *__restrict__ live,
                   int from) {
    const int slot = find_entry(start, ne, blockIdx.x);
    const BatchLevel &L = E[ids[slot]];
    if (!live[L.cand]) return;
    const int local = (int)blockIdx.x - start[slot];
    RestrictView R{};
    R.nx = (int)L.nx;
    R.ny = (int)L.ny;
    R.ncx = (int)L.F.ncx;
    R.ncy = (int)L.F.ncy;
    R.n = L.n;
    R.c4 = L.F.c4;
    R.diag = L.F.diag;
    R.a9 = L.F.a9;
    R.weight = L.F.weight;
    R.active = L.active;
    R.x = from ? L.x2 : L.x;
    R.b = L.b;
    R.bc = L.bc;
    const int tiles_y = (R.ncy + kRestrictY - 1) / kRestrictY;
    const int bx = local / tiles_y;
    restrict_tile<NINE, true>(R, bx, local - bx * tiles_y);
}

// Every candidate's coarse levels, one block each.
__global__ void __launch_bounds__(kTailThreads, 1)
    batch_tail(const BatchTail *__restrict__ T, const int *__restrict__ ids,
               const uint8_t *__restrict__ live) {
    const BatchTail &t = T[ids[blockIdx.x]];
    if (!live[t.cand]) return;
    vcycle_tail_run<true>(t.levels, t.plans, t.count, t.image, t.words, t.doubles, t.ints, t.inv,
                          t.sweeps);
}

// The per-block partial sums of the finest levels' squares: part[2 block + q].
__device__ __forceinline__ void block_sums(double a, double b, double *__restrict__ part) {
    __shared__ double sa[kBatchThreads / 32], sb[kBatchThreads / 32];
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, off);
        b += __shfl_down_sync(0xffffffffu, b, off);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        sa[warp] = a;
        sb[warp] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0.0, tb = 0.0;
        for (int w = 0; w < kBatchThreads / 32; ++w) {
            ta += sa[w];
            tb += sb[w];
        }
        part[2 * blockIdx.x] = ta;
        part[2 * blockIdx.x + 1] = tb;
    }
}

// The right-hand side and the held potentials (prepare), then r0 = b - A phi (a second
// launch: it reads the neighbours' held values).
__global__ void batch_prepare(const BatchFine *__restrict__ E, const int *__restrict__ ids,
                              const int *__restrict__ start,
                              int ne, const uint8_t *__restrict__ live) {
    const int slot = find_entry(start, ne, blockIdx.x);
    const BatchFine &F = E[ids[slot]];
    if (!live[F.cand]) return;
    const i64 f = ((i64)blockIdx.x - start[slot]) * kBatchThreads + threadIdx.x;
    if (f >= F.n) return;
    if (F.active[f]) {
        F.b[f] = (F.rho ? F.rho[f] / kEps0 : 0.0) + F.src[f];
    } else {
        F.b[f] = 0.0;
        F.phi[f] = F.value[f];
    }
}

// r0 = b - A phi, the V-cycle's first input r0, d = 0; the partial sums of |b|^2, |r0|^2.
__global__ void batch_initial(const BatchFine *__restrict__ E, const int *__restrict__ ids,
                              const int *__restrict__ start,
                              int ne, const uint8_t *__restrict__ live, double *__restrict__ part) {
    const int slot = find_entry(start, ne, blockIdx.x);
    const BatchFine &F = E[ids[slot]];
    if (!live[F.cand]) return;
    const i64 f = ((i64)blockIdx.x - start[slot]) * kBatchThreads + threadIdx.x;
    double bb = 0.0, rr = 0.0;
    if (f < F.n) {
        const double r = apply5_item(f, F.nx, F.ny, F.c4, F.diag, F.active, F.phi, F.b, F.r0);
        F.vb[f] = r;
        F.d[f] = 0.0;
        const double b = F.b[f];
        bb = b * b;
        rr = r * r;
    }
    block_sums(bb, rr, part);
}

// d += the V-cycle's correction.
__global__ void batch_correct(const BatchFine *__restrict__ E, const int *__restrict__ ids,
                              const int *__restrict__ start,
                              int ne, const uint8_t *__restrict__ live) {
    const int slot = find_entry(start, ne, blockIdx.x);
    const BatchFine &F = E[ids[slot]];
    if (!live[F.cand]) return;
    const i64 f = ((i64)blockIdx.x - start[slot]) * kBatchThreads + threadIdx.x;
    if (f < F.n) F.d[f] += F.vx[f];
}

// The true residual r = r0 - A d as the next V-cycle's input; the partial sums of |r|^2.
__global__ void batch_residual0(const BatchFine *__restrict__ E, const int *__restrict__ ids,
                              const int *__restrict__ start,
                                int ne, const uint8_t *__restrict__ live,
                                double *__restrict__ part) {
    const int slot = find_entry(start, ne, blockIdx.x);
    const BatchFine &F = E[ids[slot]];
    if (!live[F.cand]) return;
    const i64 f = ((i64)blockIdx.x - start[slot]) * kBatchThreads + threadIdx.x;
    double rr = 0.0;
    if (f < F.n) {
        const double r = apply5_item(f, F.nx, F.ny, F.c4, F.diag, F.active, F.d, F.r0, F.vb);
        rr = r * r;
    }
    block_sums(rr, 0.0, part);
}

// phi += d.
__global__ void batch_finish(const BatchFine *__restrict__ E, const int *__restrict__ ids,
                              const int *__restrict__ start,
                             int ne, const uint8_t *__restrict__ solving) {
    const int slot = find_entry(start, ne, blockIdx.x);
    const BatchFine &F = E[ids[slot]];
    if (!solving[F.cand]) return;
    const i64 f = ((i64)blockIdx.x - start[slot]) * kBatchThreads + threadIdx.x;
    if (f < F.n) F.phi[f] += F.d[f];
}

// Per live candidate (a warp each): its blocks' partial sums added in block order.  First
// call (cycle 0): the goal tol max(|b|, |r0|) and the first residual; later: the residual
// after the cycle, and whether the candidate stops -- at the goal, or after three cycles
// that did not halve its best residual (its rounding floor).  state[4 e ..]: goal, best,
// last residual, cycles without halving; cycles[e]: the cycles it ran.
__global__ void batch_check(const BatchFine *__restrict__ E, const int *__restrict__ ids,
                              const int *__restrict__ start,
                            int ne, const double *__restrict__ part, double tol, int cycle,
                            uint8_t *__restrict__ live, double *__restrict__ state,
                            int32_t *__restrict__ cycles, int32_t *__restrict__ remaining) {
    const int slot = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (slot >= ne) return;
    const int e = ids[slot];
    const BatchFine &F = E[e];
    if (!live[F.cand]) return;
    const int b0 = start[slot];
    const int b1 = slot + 1 < ne ? start[slot + 1] : b0 + (int)((F.n + kBatchThreads - 1) / kBatchThreads);
    double s0 = 0.0, s1 = 0.0;
    for (int k = b0 + lane; k < b1; k += 32) {
        s0 += part[2 * k];
        s1 += part[2 * k + 1];
    }
    for (int off = 16; off > 0; off >>= 1) {
        s0 += __shfl_down_sync(0xffffffffu, s0, off);
        s1 += __shfl_down_sync(0xffffffffu, s1, off);
    }
    if (lane != 0) return;
    double *st = state + 4 * e;
    if (cycle == 0) {
        const double scale = fmax(sqrt(s0), sqrt(s1));
        const double r = sqrt(s1);
        st[0] = tol * (scale > 0.0 ? scale : 1.0);
        st[1] = r;
        st[2] = r;
        st[3] = 0.0;
        cycles[e] = 0;
        if (!(r > st[0])) {
            live[F.cand] = 0;
            atomicSub(remaining, 1);
        }
        return;
    }
    const double r = sqrt(s0);
    cycles[e] = cycle;
    st[2] = r;
    if (r < 0.5 * st[1]) {
        st[1] = r;
        st[3] = 0.0;
    } else {
        st[3] += 1.0;
    }
    if (!(r > st[0]) || st[3] >= 3.0 || r != r) {
        live[F.cand] = 0;
        atomicSub(remaining, 1);
    }
}

}  // namespace
}  // namespace bt


struct bt_poisson_batch {
    bt_ctx *ctx = nullptr;
    std::vector<bt_poisson *> solvers;
    std::vector<i64> offset;  // each candidate's first node in the batch's arrays
    int steps = 0;            // level steps above the tails
    // A level step: all its entries (device) with their candidates and block counts (host),
    // and the launch tables of the entries whose candidates are live: their numbers and,
    // per kind of launch, each one's first block.
    struct Step {
        bt::Buffer entries;
        std::vector<int> cand, nx, ny, coarse;
        bt::Buffer ids, smooth_start, coarse_start;
        int n = 0, smooth_blocks = 0, coarse_blocks = 0;
    };
    std::vector<Step> level;
    bt::Buffer tails, tail_ids;  // one block per live candidate
    int n_tails = 0;
    size_t tail_smem = 0;
    bt::Buffer fine, fine_ids, fine_start;
    std::vector<bt::BatchFine> fine_host;  // the device table's copy
    std::vector<int> fine_nodes;           // blocks of each candidate's finest level
    int n_fine = 0, fine_blocks = 0;
    std::vector<uint8_t> compacted;        // the live set of the launch tables
    bt::Buffer live, solving, part, state, cycles, remaining;
    bt::HostBuffer host;
    int fine_sweeps = 2, coarse_sweeps = 2;
    // The smoothing tiles (interior nodes along x and y) of level 0 and of the 9-point
    // levels, and the launches a 9-point smoothing is split into (1 or 2); chosen by timing
    // at the first solve unless set (tuned == false: still to be chosen).
    int tile5[2] = {32, 32}, tile9[2] = {16, 32}, split9 = 1;
    bool tuned = false;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    ~bt_poisson_batch() {
        for (auto &e : ev)
            if (e) cudaEventDestroy(e);
    }
};

namespace bt {
namespace {

template <class T>
void upload(Buffer &dst, const std::vector<T> &src, cudaStream_t st) {
    if (src.empty()) return;
    BT_CUDA(cudaMemcpyAsync(dst.as<T>(src.size()), src.data(), sizeof(T) * src.size(),
                            cudaMemcpyHostToDevice, st));
}

// The launch tables of the candidates flagged in `alive` (host): the finished ones launch
// no blocks.  Queued on the stream, after the launches that read the old tables.
void compact(bt_poisson_batch *B, const uint8_t *alive) {
    cudaStream_t st = B->ctx->stream;
    const int count = (int)B->solvers.size();
    for (auto &S : B->level) {
        std::vector<int> ids, smooth, coarse;
        int sb = 0, cb = 0;
        const bool five = &S == &B->level[0];
        const int tx = five ? B->tile5[0] : B->tile9[0], ty = five ? B->tile5[1] : B->tile9[1];
        for (int e = 0; e < (int)S.cand.size(); ++e) {
            if (!alive[S.cand[e]]) continue;
            ids.push_back(e);
            smooth.push_back(sb);
            coarse.push_back(cb);
            sb += ((S.nx[e] + tx - 1) / tx) * ((S.ny[e] + ty - 1) / ty);
            cb += S.coarse[e];
        }
        S.n = (int)ids.size();
        S.smooth_blocks = sb;
        S.coarse_blocks = cb;
        upload(S.ids, ids, st);
        upload(S.smooth_start, smooth, st);
        upload(S.coarse_start, coarse, st);
    }
    std::vector<int> tails, fine, start;
    int fb = 0;
    for (int c = 0; c < count; ++c) {
        if (!alive[c]) continue;
        tails.push_back(c);
        fine.push_back(c);
        start.push_back(fb);
        fb += B->fine_nodes[c];
    }
    B->n_tails = (int)tails.size();
    B->n_fine = (int)fine.size();
    B->fine_blocks = fb;
    upload(B->tail_ids, tails, st);
    upload(B->fine_ids, fine, st);
    upload(B->fine_start, start, st);
    B->compacted.assign(alive, alive + count);
}

// The staged smoother's nodes a thread per colour for a tile (tx, ty) and `count` phases.
int stage_own(bool nine, int tx, int ty, int count) {
    const int halo = stage_halo(count);
    const int per = (tx + 2 * halo) * (ty + 2 * halo) / (nine ? 4 : 2);
    return (per + kStageThreads - 1) / kStageThreads;
}

int fine_own(int count) { return stage_own(false, kStage5X, kStage5Y, count); }

Phases batch_phases(int sweeps, int colours, bool pre, int first, int count) {
    Phases ph{};
    std::vector<int> order;
    for (int s = 0; s < sweeps; ++s)
        for (int c = 0; c < colours; ++c) order.push_back(pre ? c : colours - 1 - c);
    ph.count = count;
    for (int k = 0; k < count; ++k) ph.colour[k] = order[first + k];
    return ph;
}

// One staged launch over step l's live entries: phases [first, first + count) of the
// smoothing, from buffer `from` into the other.
void batch_smooth_launch(bt_poisson_batch *B, int l, bool pre, int first, int count, int from,
                         int prolong, int zero_in) {
    bt_ctx *ctx = B->ctx;
    auto &S = B->level[l];
    const bool nine = l > 0;
    const uint8_t *live = B->live.as<uint8_t>(B->solvers.size());
    const BatchLevel *E = S.entries.as<BatchLevel>(S.cand.size());
    const int *ids = S.ids.as<int>(S.n), *start = S.smooth_start.as<int>(S.n);
    const int tx = nine ? B->tile9[0] : B->tile5[0], ty = nine ? B->tile9[1] : B->tile5[1];
    // the register form for the tiles of the tuner's list
#define BT_BATCH_TILE(N, X, Y, C)                                                              \
    if (nine == N && tx == X && ty == Y && count == C && first % (N ? 4 : 2) == 0) {             \
        if (pre)                                                                                   \
            BT_LAUNCH(ctx, (batch_smooth_tile<N, X, Y, C, false>), S.smooth_blocks,                \
                      (Tile<N, X, Y, C>::threads), 0, ctx->stream, E, ids, start, S.n, live, from, \
                      prolong, zero_in);                                                           \
        else                                                                                       \
            BT_LAUNCH(ctx, (batch_smooth_tile<N, X, Y, C, true>), S.smooth_blocks,                 \
                      (Tile<N, X, Y, C>::threads), 0, ctx->stream, E, ids, start, S.n, live, from, \
                      prolong, zero_in);                                                           \
        return;                                                                                    \
    }
    BT_BATCH_TILE(false, 32, 32, 4)
    BT_BATCH_TILE(false, 32, 16, 4)
    BT_BATCH_TILE(false, 16, 32, 4)
    BT_BATCH_TILE(false, 64, 16, 4)
    BT_BATCH_TILE(true, 16, 32, 8)
    BT_BATCH_TILE(true, 16, 32, 4)
    BT_BATCH_TILE(true, 16, 16, 4)
    BT_BATCH_TILE(true, 32, 16, 4)
    BT_BATCH_TILE(true, 32, 32, 4)
#undef BT_BATCH_TILE
    const Phases ph = batch_phases(nine ? B->coarse_sweeps : B->fine_sweeps, nine ? 4 : 2, pre,
                                   first, count);
    const size_t smem = stage_smem(nine, tx, ty, stage_halo(count));
    const int own = stage_own(nine, tx, ty, count);
#define BT_BATCH_SMOOTH(N, R)                                                                 \
    BT_LAUNCH(ctx, (batch_smooth<N, R>), S.smooth_blocks, kStageThreads, smem, ctx->stream, E, \
              ids, start, S.n, live, tx, ty, ph, from, prolong, zero_in)
    if (!nine && own == 1)
        BT_BATCH_SMOOTH(false, 1);
    else if (!nine && own == 2)
        BT_BATCH_SMOOTH(false, 2);
    else if (!nine && own == 3)
        BT_BATCH_SMOOTH(false, 3);
    else if (nine && own == 1)
        BT_BATCH_SMOOTH(true, 1);
    else if (nine && own == 2)
        BT_BATCH_SMOOTH(true, 2);
    else
        BT_REQUIRE(false, "poisson batch: a smoothing tile too large for its block");
#undef BT_BATCH_SMOOTH
}

// The smoothing of step l's live entries before (pre) or after the coarse correction;
// returns the buffer that holds the result (0: x, 1: x2).  The pre-smoothing starts from
// zero; the post-smoothing adds the prolonged correction as it reads.  Before the
// correction the input is the pre-smoothing's result `from`.
int batch_smooth_step(bt_poisson_batch *B, int l, bool pre, int from = 0) {
    auto &S = B->level[l];
    if (S.n == 0) return from;
    const bool nine = l > 0;
    const int phases = nine ? 4 * B->coarse_sweeps : 2 * B->fine_sweeps;
    const int split = nine ? B->split9 : 1;
    const int per = (phases + split - 1) / split;
    int in = pre ? 0 : from;
    for (int first = 0, k = 0; first < phases; first += per, ++k) {
        const int count = std::min(per, phases - first);
        batch_smooth_launch(B, l, pre, first, count, in, (!pre && k == 0) ? 1 : 0,
                            (pre && k == 0) ? 1 : 0);
        in ^= 1;
    }
    return in;
}

// One V-cycle of every live candidate: level 0's b (its residual) into level 0's x.
void batch_vcycle(bt_poisson_batch *B) {
    bt_ctx *ctx = B->ctx;
    cudaStream_t st = ctx->stream;
    const uint8_t *live = B->live.as<uint8_t>(B->solvers.size());
    std::vector<int> held(B->steps, 0);  // where each step's pre-smoothing left x
    for (int l = 0; l < B->steps; ++l) {
        auto &S = B->level[l];
        if (S.n == 0) continue;
        const BatchLevel *E = S.entries.as<BatchLevel>(S.cand.size());
        const int *ids = S.ids.as<int>(S.n);
        held[l] = batch_smooth_step(B, l, true);
        if (l == 0)
            BT_LAUNCH(ctx, batch_restrict<false>, S.coarse_blocks, kRestrictThreads, 0, st, E, ids,
                      S.coarse_start.as<int>(S.n), S.n, live, held[l]);
        else
            BT_LAUNCH(ctx, batch_restrict<true>, S.coarse_blocks, kRestrictThreads, 0, st, E, ids,
                      S.coarse_start.as<int>(S.n), S.n, live, held[l]);
    }
    if (B->n_tails)
        BT_LAUNCH(ctx, batch_tail, (unsigned)B->n_tails, kTailThreads, B->tail_smem, st,
                  B->tails.as<BatchTail>(B->solvers.size()), B->tail_ids.as<int>(B->n_tails),
                  live);
    for (int l = B->steps - 1; l >= 0; --l) {
        // the post-smoothing must leave x in the level's x buffer (the next coarser level's
        // x, or level 0's output)
        const int at = batch_smooth_step(B, l, false, held[l]);
        BT_REQUIRE(B->level[l].n == 0 || at == 0, "poisson batch: smoothing left x in x2");
    }
    BT_CHECK_LAUNCH();
}

}  // namespace
}  // namespace bt

namespace bt {
namespace {

// The project's autotuner of the batched V-cycle: the staged smoothing tiles of level 0 and
// of the 9-point levels (and whether a 9-point smoothing is one launch of all its phases,
// with a halo as wide as them, or two of half as many), timed on this batch's own V-cycle
// (two cycles each, CUDA events on the stream) from the residual of its first solve; the
// fastest is kept.  The choices trade a tile's re-read halo against blocks per SM.
void tune_tiling(bt_poisson_batch *B) {
    cudaStream_t st = B->ctx->stream;
    const std::vector<uint8_t> set = B->compacted;
    auto time_cycle = [&]() {
        compact(B, set.data());
        BT_CUDA(cudaEventRecord(B->ev[0], st));
        for (int k = 0; k < 2; ++k) batch_vcycle(B);
        BT_CUDA(cudaEventRecord(B->ev[1], st));
        BT_CUDA(cudaEventSynchronize(B->ev[1]));
        float ms = 0.0f;
        BT_CUDA(cudaEventElapsedTime(&ms, B->ev[0], B->ev[1]));
        return ms;
    };
    const int tiles5[][2] = {{32, 32}, {32, 16}, {16, 32}, {64, 16}};
    float best = 1e30f;
    int pick5[2] = {B->tile5[0], B->tile5[1]};
    for (const auto &t : tiles5) {
        if (stage_own(false, t[0], t[1], 2 * B->fine_sweeps) > 3) continue;
        B->tile5[0] = t[0];
        B->tile5[1] = t[1];
        const float ms = time_cycle();
        if (ms < best) {
            best = ms;
            pick5[0] = t[0];
            pick5[1] = t[1];
        }
    }
    B->tile5[0] = pick5[0];
    B->tile5[1] = pick5[1];
    const int tiles9[][3] = {{16, 32, 1}, {16, 32, 2}, {16, 16, 2}, {32, 16, 2}, {32, 32, 2}};
    best = 1e30f;
    int pick9[3] = {B->tile9[0], B->tile9[1], B->split9};
    for (const auto &t : tiles9) {
        const int phases = 4 * B->coarse_sweeps;
        const int count = (phases + t[2] - 1) / t[2];
        if (stage_own(true, t[0], t[1], count) > 2 ||
            stage_smem(true, t[0], t[1], stage_halo(count)) > 200 * 1024)
            continue;
        B->tile9[0] = t[0];
        B->tile9[1] = t[1];
        B->split9 = t[2];
        const float ms = time_cycle();
        if (ms < best) {
            best = ms;
            pick9[0] = t[0];
            pick9[1] = t[1];
            pick9[2] = t[2];
        }
    }
    B->tile9[0] = pick9[0];
    B->tile9[1] = pick9[1];
    B->split9 = pick9[2];
    compact(B, set.data());
    B->tuned = true;
}

}  // namespace
}  // namespace bt

extern "C" int bt_poisson_batch_create(bt_ctx *ctx, bt_poisson *const *solvers, int64_t count,
                                       const int64_t *offset, bt_poisson_batch **out) {
    return bt::guarded([&] {
        BT_REQUIRE(ctx && solvers && offset && out, "poisson batch: null argument");
        BT_REQUIRE(count >= 1 && count <= (1 << 20), "poisson batch: 1 to 2^20 candidates");
        auto B = new bt_poisson_batch;
        try {
            B->ctx = ctx;
            cudaStream_t st = ctx->stream;
            B->solvers.assign(solvers, solvers + count);
            B->offset.assign(offset, offset + count);
            bt_poisson *first = B->solvers[0];
            BT_REQUIRE(first, "poisson batch: null solver");
            B->fine_sweeps = first->fine_sweeps;
            B->coarse_sweeps = first->coarse_sweeps;
            for (i64 c = 0; c < count; ++c) {
                bt_poisson *p = B->solvers[c];
                BT_REQUIRE(p, "poisson batch: null solver");
                BT_REQUIRE(p->ctx == ctx, "poisson batch: every solver must share the context");
                BT_REQUIRE(!p->transposed, "poisson batch: the transposed solver is not batched");
                BT_REQUIRE(p->staged, "poisson batch: needs the staged smoother");
                BT_REQUIRE(p->fine_sweeps == B->fine_sweeps && p->coarse_sweeps == B->coarse_sweeps,
                           "poisson batch: every solver needs the same smoothing sweeps");
                BT_REQUIRE(B->coarse_sweeps * 4 <= bt::kMaxPhases && B->fine_sweeps * 2 <= bt::kMaxPhases,
                           "poisson batch: a smoothing must fit one staged launch");
                BT_REQUIRE(bt::fine_own(2 * B->fine_sweeps) <= 3,
                           "poisson batch: the fine smoothing tile is too large for its block");
                BT_REQUIRE(p->tail_start >= 1,
                           "poisson batch: a candidate's mesh is too small for the batched cycle");
                B->steps = std::max(B->steps, p->tail_start);
                B->tail_smem = std::max(B->tail_smem, p->tail_smem);
            }
            B->level.resize(B->steps);
            for (int l = 0; l < B->steps; ++l) {
                std::vector<bt::BatchLevel> E;
                auto &S = B->level[l];
                const bool five = l == 0;
                for (i64 c = 0; c < count; ++c) {
                    bt_poisson *p = B->solvers[c];
                    if (l >= p->tail_start) continue;
                    bt::Level &L = p->levels[l], &C = p->levels[l + 1];
                    bt::BatchLevel e{};
                    e.cand = (int)c;
                    e.nx = L.nx;
                    e.ny = L.ny;
                    e.n = L.n;
                    if (five) {
                        e.c4 = L.c4.as<double>(4 * L.n);
                        e.diag = L.diag.as<double>(L.n);
                    } else {
                        e.a9 = L.a9.as<double>(9 * L.n);
                    }
                    e.active = L.active.as<uint8_t>(L.n);
                    e.x = L.x.as<double>(L.n);
                    e.x2 = L.x2.as<double>(L.n);
                    e.b = L.b.as<double>(L.n);
                    e.F = bt::fine_of(L, C, five);
                    e.xc = C.x.as<double>(C.n);
                    e.bc = C.b.as<double>(C.n);
                    E.push_back(e);
                    S.cand.push_back((int)c);
                    S.nx.push_back((int)L.nx);
                    S.ny.push_back((int)L.ny);
                    S.coarse.push_back((int)(((C.nx + bt::kRestrictX - 1) / bt::kRestrictX) *
                                             ((C.ny + bt::kRestrictY - 1) / bt::kRestrictY)));
                }
                bt::upload(S.entries, E, st);
            }
            std::vector<bt::BatchTail> T;
            std::vector<bt::BatchFine> F;
            int all_blocks = 0;
            for (i64 c = 0; c < count; ++c) {
                bt_poisson *p = B->solvers[c];
                const int first_tail = p->tail_start;
                const int levels = (int)p->levels.size();
                const bt::Level &Lc = p->levels.back();
                bt::BatchTail t{};
                t.cand = (int)c;
                t.levels = p->tail_levels.as<bt::TailLevel>(levels - first_tail);
                t.plans = p->tail_plans.as<bt::TailPlan>(levels - first_tail);
                t.count = levels - first_tail;
                t.image = static_cast<const uint4 *>(p->tail_image.get(16 * (size_t)p->tail_words));
                t.words = p->tail_words;
                t.doubles = p->tail_doubles;
                t.ints = p->tail_ints;
                t.inv = p->inv.as<double>(Lc.n * Lc.n);
                t.sweeps = p->coarse_sweeps;
                T.push_back(t);
                bt::Level &L0 = p->levels[0];
                const i64 n = p->n;
                bt::BatchFine f{};
                f.cand = (int)c;
                f.nx = p->nx;
                f.ny = p->ny;
                f.n = n;
                f.c4 = L0.c4.as<double>(4 * n);
                f.diag = L0.diag.as<double>(n);
                f.src = p->src.as<double>(n);
                f.value = p->value_eff.as<double>(n);
                f.active = L0.active.as<uint8_t>(n);
                f.b = p->rhs.as<double>(n);
                f.r0 = p->r0.as<double>(n);
                f.d = p->delta.as<double>(n);
                f.vb = L0.b.as<double>(n);
                f.vx = L0.x.as<double>(n);
                F.push_back(f);
                B->fine_nodes.push_back((int)bt::blocks_for(n, bt::kBatchThreads));
                all_blocks += B->fine_nodes.back();
            }
            B->fine_host = F;
            bt::upload(B->tails, T, st);
            bt::upload(B->fine, F, st);
            {
                // the largest staged tile the tuner tries (bt::tune_tiling)
                const int big = 200 * 1024;
                BT_CUDA(cudaFuncSetAttribute(bt::batch_smooth<false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
                BT_CUDA(cudaFuncSetAttribute(bt::batch_smooth<false, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
                BT_CUDA(cudaFuncSetAttribute(bt::batch_smooth<false, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
                BT_CUDA(cudaFuncSetAttribute(bt::batch_smooth<true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
                BT_CUDA(cudaFuncSetAttribute(bt::batch_smooth<true, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
                BT_CUDA(cudaFuncSetAttribute(bt::batch_tail, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)bt::kTailSmemMax));
            }
            for (auto &e : B->ev) BT_CUDA(cudaEventCreate(&e));
            B->live.as<uint8_t>(count);
            B->solving.as<uint8_t>(count);
            B->part.as<double>(2 * (size_t)all_blocks);
            B->state.as<double>(4 * (size_t)count);
            B->cycles.as<int32_t>(count);
            B->remaining.as<int32_t>(1);
            BT_CUDA(cudaStreamSynchronize(st));
        } catch (...) {
            delete B;
            throw;
        }
        *out = B;
    });
}

extern "C" int bt_poisson_batch_destroy(bt_poisson_batch *B) {
    return bt::guarded([&] {
        if (!B) return;
        cudaStreamSynchronize(B->ctx->stream);
        delete B;
    });
}

extern "C" int bt_poisson_batch_solve(bt_poisson_batch *B, double *phi, const double *rho,
                                      const uint8_t *members, double tol, int32_t max_cycles,
                                      int32_t *cycles, double *residual) {
    return bt::guarded([&] {
        BT_REQUIRE(B && phi && members, "poisson batch: null argument");
        BT_REQUIRE(tol > 0.0, "poisson batch: the tolerance must be positive");
        BT_REQUIRE(max_cycles >= 1, "poisson batch: max_cycles must be positive");
        bt_ctx *ctx = B->ctx;
        cudaStream_t st = ctx->stream;
        const i64 count = (i64)B->solvers.size();
        bt::Timed timed(ctx, "field_solve");
        // every member's hierarchy of its plain operator
        int members_n = 0;
        for (i64 c = 0; c < count; ++c) {
            if (!members[c]) continue;
            ++members_n;
            bt_poisson *p = B->solvers[c];
            if (!p->built || p->reaction_on) bt::build_hierarchy(p, nullptr);
        }
        if (members_n == 0) return;
        {
            // point the finest entries at this call's potential and density
            std::vector<bt::BatchFine> &F = B->fine_host;
            bool moved = false;
            for (i64 c = 0; c < count; ++c) {
                double *ph = phi + B->offset[c];
                const double *rh = rho ? rho + B->offset[c] : nullptr;
                if (F[c].phi != ph || F[c].rho != rh) moved = true;
                F[c].phi = ph;
                F[c].rho = rh;
            }
            if (moved) bt::upload(B->fine, F, st);
        }
        uint8_t *live = B->live.as<uint8_t>(count);
        uint8_t *solving = B->solving.as<uint8_t>(count);
        BT_CUDA(cudaMemcpyAsync(live, members, count, cudaMemcpyHostToDevice, st));
        BT_CUDA(cudaMemcpyAsync(solving, members, count, cudaMemcpyHostToDevice, st));
        int32_t *remaining = B->remaining.as<int32_t>(1);
        uint8_t *flags = static_cast<uint8_t *>(B->host.get((size_t)count + 64));
        int32_t *host_remaining = reinterpret_cast<int32_t *>(flags + ((count + 15) / 16) * 16);
        *host_remaining = members_n;
        BT_CUDA(cudaMemcpyAsync(remaining, host_remaining, sizeof(int32_t), cudaMemcpyHostToDevice, st));
        bt::compact(B, members);
        const bt::BatchFine *F = B->fine.as<bt::BatchFine>(count);
        double *part = B->part.as<double>(1);
        double *state = B->state.as<double>(4 * (size_t)count);
        int32_t *cyc = B->cycles.as<int32_t>(count);
        const int T = bt::kBatchThreads;
        auto fine_launch = [&](auto kernel, auto... more) {
            if (B->fine_blocks)
                BT_LAUNCH(ctx, kernel, B->fine_blocks, T, 0, st, F, B->fine_ids.as<int>(B->n_fine),
                          B->fine_start.as<int>(B->n_fine), B->n_fine, more...);
        };
        auto check = [&](int cycle) {
            BT_LAUNCH(ctx, bt::batch_check, bt::blocks_for((i64)B->n_fine * 32, 256), 256, 0, st, F,
                      B->fine_ids.as<int>(B->n_fine), B->fine_start.as<int>(B->n_fine),
                      B->n_fine, (const double *)part, tol, cycle, live, state, cyc, remaining);
        };
        fine_launch(bt::batch_prepare, (const uint8_t *)live);
        fine_launch(bt::batch_initial, (const uint8_t *)live, part);
        check(0);
        BT_CHECK_LAUNCH();
        if (!B->tuned) bt::tune_tiling(B);
        for (int cycle = 1; cycle <= max_cycles; ++cycle) {
            BT_CUDA(cudaMemcpyAsync(flags, live, count, cudaMemcpyDeviceToHost, st));
            BT_CUDA(cudaStreamSynchronize(st));
            int alive = 0, before = 0;
            for (i64 c = 0; c < count; ++c) {
                alive += flags[c] != 0;
                before += B->compacted[c] != 0;
            }
            if (alive == 0) break;
            // launch tables of the live candidates only, once enough of them have finished
            if (10 * alive <= 9 * before) bt::compact(B, flags);
            {
                bt::Timed vt(ctx, "vcycle");
                bt::batch_vcycle(B);
            }
            fine_launch(bt::batch_correct, (const uint8_t *)live);
            fine_launch(bt::batch_residual0, (const uint8_t *)live, part);
            check(cycle);
            BT_CHECK_LAUNCH();
        }
        bt::compact(B, members);
        fine_launch(bt::batch_finish, (const uint8_t *)solving);
        BT_CHECK_LAUNCH();
        std::vector<double> S(4 * count);
        std::vector<int32_t> C(count);
        BT_CUDA(cudaMemcpyAsync(S.data(), state, sizeof(double) * 4 * count, cudaMemcpyDeviceToHost, st));
        BT_CUDA(cudaMemcpyAsync(C.data(), cyc, sizeof(int32_t) * count, cudaMemcpyDeviceToHost, st));
        BT_CUDA(cudaStreamSynchronize(st));
        for (i64 c = 0; c < count; ++c) {
            if (!members[c]) continue;
            if (cycles) cycles[c] = C[c];
            if (residual) residual[c] = S[4 * c + 2];
            // a residual stalled within 1e4 of the goal is the floor of its own rounding (an
            // infinite one meets its own relative goal)
            if (!(S[4 * c + 2] <= 1e4 * S[4 * c]) || !std::isfinite(S[4 * c + 2]))
                throw bt::Error{BT_ERR_NOCONV, "batched field solve: a candidate did not reach the tolerance"};
        }
    });
}

extern "C" int bt_poisson_batch_tiling(bt_poisson_batch *B, int32_t set, int32_t *tiling) {
    return bt::guarded([&] {
        BT_REQUIRE(B && tiling, "poisson batch: null argument");
        if (set) {
            if (tiling[0] <= 0) {
                B->tuned = false;
                return;
            }
            for (int q = 0; q < 5; ++q)
                BT_REQUIRE(tiling[q] > 0, "poisson batch: tile sizes and split must be positive");
            BT_REQUIRE(tiling[4] <= 2, "poisson batch: a 9-point smoothing splits into 1 or 2 launches");
            const int phases9 = 4 * B->coarse_sweeps, count9 = (phases9 + tiling[4] - 1) / tiling[4];
            BT_REQUIRE(bt::stage_own(false, tiling[0], tiling[1], 2 * B->fine_sweeps) <= 3 &&
                           bt::stage_smem(false, tiling[0], tiling[1], bt::stage_halo(2 * B->fine_sweeps)) <= 200 * 1024,
                       "poisson batch: the level-0 tile is too large for its block");
            BT_REQUIRE(bt::stage_own(true, tiling[2], tiling[3], count9) <= 2 &&
                           bt::stage_smem(true, tiling[2], tiling[3], bt::stage_halo(count9)) <= 200 * 1024,
                       "poisson batch: the 9-point tile is too large for its block");
            B->tile5[0] = tiling[0];
            B->tile5[1] = tiling[1];
            B->tile9[0] = tiling[2];
            B->tile9[1] = tiling[3];
            B->split9 = tiling[4];
            B->tuned = true;
            return;
        }
        tiling[0] = B->tile5[0];
        tiling[1] = B->tile5[1];
        tiling[2] = B->tile9[0];
        tiling[3] = B->tile9[1];
        tiling[4] = B->split9;
        tiling[5] = B->tuned ? 1 : 0;
    });
}

extern "C" int bt_poisson_set_context(bt_poisson *p, bt_ctx *ctx) {
    return bt::guarded([&] {
        BT_REQUIRE(p && ctx, "poisson: null argument");
        if (p->ctx == ctx) return;
        BT_REQUIRE(p->ctx->device == ctx->device, "poisson: the new context is on another device");
        // the old context's queued work first; its captured V-cycle is its own
        BT_CUDA(cudaStreamSynchronize(p->ctx->stream));
        bt::drop_graphs(p);
        p->ctx = ctx;
    });
}
