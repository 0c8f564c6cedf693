// mg.cu — an aggregation multigrid V-cycle as the preconditioner of the
// mixed form's pressure solve (RT_OPT_MIXED_PRECOND -2) and momentum solve
// (RT_OPT_MIXED_PRECOND_U -2) on structured meshes, in FP32.
//
// The matrix of a structured mesh is a 7-point stencil on the box
// (nx x ny x nz, inactive box cells outside the mesh).  Its coefficients are
// formed in box order, level by level: the diagonal and, for each of the i-1, j-1 and
// k-1 neighbours c' of a cell c, A[c][c'] (xl, yl, zl) and A[c'][c] (xu,
// yu, zu); a zero diagonal marks an inactive cell.  The symmetric pressure
// matrix keeps one copy (the u arrays alias the l arrays).  A coarse level
// aggregates 2 x 2 x 2 cells (a direction of one cell is not coarsened) with
// piecewise-constant prolongation P and restriction P^T, so its operator
// P^T A P is again a 7-point stencil: the children's diagonals plus both
// couplings of every child pair inside the aggregate, and the sums of the
// children's couplings across each aggregate face.  Levels are added until
// the box has at most kCoarse cells; that last one is smoothed by one CTA.
//
// One application (a V-cycle from x = 0): on every level kNu red-black
// Gauss-Seidel sweeps (red then black), the residual restricted into the
// next level's right-hand side; on the coarsest level kCoarseSweeps
// symmetric sweeps; on the way up the correction prolongated (scaled by
// kOver, over-correction for the unsmoothed aggregation) and kNu sweeps in
// the reverse order (black then red).  kNu and kOver were chosen on the
// 1M-cell contraction's pressure solve: (1, 1.6) 331 iterations, (2, 1.6)
// 185, (1, 1.9) 382, (2, 1.3) 162, (2, 1.0) 140, (3, 1.3) 108.  On a
// symmetric matrix the smoother and its adjoint, and a constant scaling,
// keep the preconditioner symmetric, as PCG needs; BiCGStab (the momentum
// solve) needs no symmetry, and the components of a vector solve go through
// one cycle together, sharing every coefficient load.
//
// The cycle's passes work on arrays split by colour: the cells of one colour of a
// row (j, k) are consecutive (i = 2 ii + o, o = (colour + j + k) % 2, at row * hx +
// ii), with the diagonal and the six couplings of a cell beside it, so that a
// half-sweep reads and writes its colour's arrays in whole lines and of the other
// colour only x; in box order it read every line of every array for half of the
// cells.  Neighbours outside the box have a zero coupling and an index inside
// the array.  Three passes of the textbook cycle are folded into others, with
// the same arithmetic on the same values: the first red half-sweep of a coarse
// level from x = 0 is b / dg, formed by the restriction; the prolongation is
// formed by the first black half-sweep after it as it reads the red values (the
// values it would leave in x are overwritten before anything else reads them);
// and level 0's last red half-sweep writes the result.
//
// What bounds it: on the 1M-cell contraction level 0 is 48 (pressure) or 69 MB
// (momentum), inside the L2, and its half-sweeps run at L2 bandwidth; the small
// levels are bound by the latency of a pass, so passes overlap their start with
// the end of the one before, and the smallest levels run in one CTA.
#include <algorithm>
#include <array>

#include "rt_internal.h"
#include "sweep.h"

namespace rt {

namespace {

constexpr int kCoarse = 512;        // cells of the level smoothed by one CTA
constexpr int kCoarseSweeps = 16;   // symmetric sweeps there
constexpr float kOver = 1.3f;       // coarse-correction scaling
constexpr int kNu = 3;              // red-black sweeps before and after the coarse correction
constexpr int kMaxLevels = 16;      // levels of a hierarchy, at most (a 2^16 box side)
constexpr int kTailCells = 4096;    // levels of at most this many box cells run in one CTA
constexpr size_t kTailSmem = 224 * 1024;   // and its shared memory
constexpr int kPassBlock = 128;

struct MgLev {
    int nx, ny, nz, n;
    int hx, nh;       // cells of one colour in a row, in the level (padded rows)
    size_t np, ns;    // strides of the box-order and of the split arrays
    float *dg, *xl, *yl, *zl, *xu, *yu, *zu;   // box order: the hierarchy's construction
    float *co;        // split: dg and the couplings to -x +x -y +y -z +z, [7][2 colours][ns]
    float *x, *b;     // split: [3 components][2 colours][ns]
};
constexpr int kBoxArrays = 7, kSplitArrays = 2 * 7 + 2 * 3 + 2 * 3;

__device__ __forceinline__ void box_ijk(const MgLev &L, int b, int &i, int &j, int &k) {
    i = b % L.nx;
    const int r = b / L.nx;
    j = r % L.ny;
    k = r / L.ny;
}

// where a colour's cell t = row * hx + ii is, and its neighbours in the other
// colour's array
struct At {
    int ii, j, k, o;
};
__device__ __forceinline__ At at_of(int nx, int ny, int hx, int colour, int t) {
    At a;
    const int row = t / hx;
    a.ii = t - row * hx;
    a.j = row % ny;
    a.k = row / ny;
    a.o = (colour + a.j + a.k) & 1;
    return a;
}
struct Nb6 {
    int i[6];
};
__device__ __forceinline__ Nb6 neighbours(int ny, int nz, int hx, const At &a, int t) {
    Nb6 n;
    n.i[0] = a.o || a.ii == 0 ? t : t - 1;
    n.i[1] = a.o && a.ii + 1 < hx ? t + 1 : t;
    n.i[2] = a.j > 0 ? t - hx : t;
    n.i[3] = a.j + 1 < ny ? t + hx : t;
    n.i[4] = a.k > 0 ? t - hx * ny : t;
    n.i[5] = a.k + 1 < nz ? t + hx * ny : t;
    return n;
}
// sum over the six neighbours of a_nb x_nb
__device__ __forceinline__ float nb_sum(const float (&c)[7], const Nb6 &n, const float *x) {
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 6; ++q) s = __fmaf_rn(c[q + 1], x[n.i[q]], s);
    return s;
}

// the components of m that still iterate (dm: a device word, or null)
__device__ __forceinline__ unsigned live(unsigned m, const unsigned *dm) { return dm ? m & *dm : m; }

// The passes of a V-cycle are launched to start while the pass before still runs
// (programmatic dependent launch): a thread loads its cell's coefficients, which
// no pass writes, and then waits until the pass before has finished.  Every pass
// waits before it touches x or b, so each starts them after all earlier ones.  The
// first lets none of the others start until it has itself waited for what came
// before the cycle, so the rest read the mask of components at once.

// level 0 from the FP64 LDU matrix (box arrays zeroed before): the face to
// the lower neighbour c' of cell c carries A[c][c'] = lower, A[c'][c] = upper
__global__ void k_mg_fine(int N, const int *__restrict__ boxOf, const int *__restrict__ faceLo,
                          const double *__restrict__ diag, const double *__restrict__ upper,
                          const double *__restrict__ lower, MgLev L, int sym) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    const int b = boxOf[c];
    L.dg[b] = (float)diag[c];
    const int fz = faceLo[c], fy = faceLo[N + c], fx = faceLo[2 * N + c];
    L.zl[b] = fz >= 0 ? (float)lower[fz] : 0.0f;
    L.yl[b] = fy >= 0 ? (float)lower[fy] : 0.0f;
    L.xl[b] = fx >= 0 ? (float)lower[fx] : 0.0f;
    if (!sym) {
        L.zu[b] = fz >= 0 ? (float)upper[fz] : 0.0f;
        L.yu[b] = fy >= 0 ? (float)upper[fy] : 0.0f;
        L.xu[b] = fx >= 0 ? (float)upper[fx] : 0.0f;
    }
}

// the Galerkin coarse operator of piecewise-constant aggregation
__global__ void k_mg_coarsen(MgLev F, MgLev C, int sym) {
    const int B = blockIdx.x * blockDim.x + threadIdx.x;
    if (B >= C.n) return;
    int I, J, K;
    box_ijk(C, B, I, J, K);
    const int fx = F.nx == C.nx ? 1 : 2, fy = F.ny == C.ny ? 1 : 2, fz = F.nz == C.nz ? 1 : 2;
    float dg = 0.0f, xl = 0.0f, yl = 0.0f, zl = 0.0f, xu = 0.0f, yu = 0.0f, zu = 0.0f;
    for (int dk = 0; dk < fz; ++dk)
        for (int dj = 0; dj < fy; ++dj)
            for (int di = 0; di < fx; ++di) {
                const int i = I * fx + di, j = J * fy + dj, k = K * fz + dk;
                if (i >= F.nx || j >= F.ny || k >= F.nz) continue;
                const int b = i + F.nx * (j + F.ny * k);
                const float d = F.dg[b];
                if (d == 0.0f) continue;   // inactive
                dg += d;
                // a coupling pair to the lower neighbour inside the aggregate
                // adds both directions to the diagonal (a_ij + a_ji), one
                // across it adds to the coarse couplings
                if (di == 1) {
                    dg += F.xl[b] + F.xu[b];
                } else {
                    xl += F.xl[b];
                    xu += F.xu[b];
                }
                if (dj == 1) {
                    dg += F.yl[b] + F.yu[b];
                } else {
                    yl += F.yl[b];
                    yu += F.yu[b];
                }
                if (dk == 1) {
                    dg += F.zl[b] + F.zu[b];
                } else {
                    zl += F.zl[b];
                    zu += F.zu[b];
                }
            }
    C.dg[B] = dg;
    C.xl[B] = I > 0 ? xl : 0.0f;
    C.yl[B] = J > 0 ? yl : 0.0f;
    C.zl[B] = K > 0 ? zl : 0.0f;
    if (!sym) {
        C.xu[B] = I > 0 ? xu : 0.0f;
        C.yu[B] = J > 0 ? yu : 0.0f;
        C.zu[B] = K > 0 ? zu : 0.0f;
    }
}

// the split coefficients of a level, once its box-order ones are complete, and x = 0
// where the diagonal is zero: no pass writes x there, and it may hold that of an
// earlier matrix in which the cell had one
__global__ void k_mg_split(MgLev L) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= 2 * L.nh) return;
    const int colour = q >= L.nh, t = q - colour * L.nh;
    const At a = at_of(L.nx, L.ny, L.hx, colour, t);
    const int i = 2 * a.ii + a.o, b = i + L.nx * (a.j + L.ny * a.k);
    float c[7] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (i < L.nx) c[0] = L.dg[b];
    if (c[0] != 0.0f) {
        const int sy = L.nx, sz = L.nx * L.ny;
        if (i > 0) c[1] = L.xl[b];
        if (i + 1 < L.nx) c[2] = L.xu[b + 1];
        if (a.j > 0) c[3] = L.yl[b];
        if (a.j + 1 < L.ny) c[4] = L.yu[b + sy];
        if (a.k > 0) c[5] = L.zl[b];
        if (a.k + 1 < L.nz) c[6] = L.zu[b + sz];
    }
#pragma unroll
    for (int k = 0; k < 7; ++k) L.co[(2 * k + colour) * L.ns + t] = c[k];
    if (c[0] == 0.0f)
#pragma unroll
        for (int q = 0; q < 3; ++q) L.x[(2 * q + colour) * L.ns + t] = 0.0f;
}

__device__ __forceinline__ void coeffs(const MgLev &L, int colour, int t, float (&c)[7]) {
#pragma unroll
    for (int k = 0; k < 7; ++k) c[k] = L.co[(2 * k + colour) * L.ns + t];
}
__device__ __forceinline__ float *split(float *a, const MgLev &L, int q, int colour) {
    return a + (2 * q + colour) * L.ns;
}

// level 0 from x = 0: the right-hand side from the residual (cell order,
// component k at k N), then the red half-sweep (x_red = b / dg); a thread the
// cells 2 ii and 2 ii + 1 of a row
template <class T>
__global__ void k_mg_first(MgLev L, const int *__restrict__ cellAt, int N, unsigned m, const T *r, const unsigned *dm) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L.nh) return;
    const At a = at_of(L.nx, L.ny, L.hx, 0, t);   // (o: the red cell's place in the pair)
    const int b0 = 2 * a.ii + L.nx * (a.j + L.ny * a.k);
    const int c0 = cellAt[b0], c1 = 2 * a.ii + 1 < L.nx ? cellAt[b0 + 1] : -1;
    const int red = a.o ? c1 : c0, black = a.o ? c0 : c1;
    wait_for_previous();
    next_may_start();
    m = live(m, dm);
    const float d = L.co[t];
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if ((m >> q) & 1u) {
            const float rr = red >= 0 ? (float)r[(size_t)q * N + red] : 0.0f;
            split(L.b, L, q, 0)[t] = rr;
            split(L.b, L, q, 1)[t] = black >= 0 ? (float)r[(size_t)q * N + black] : 0.0f;
            split(L.x, L, q, 0)[t] = d != 0.0f ? rr / d : 0.0f;
        }
}

// one half-sweep of red-black Gauss-Seidel (colour 0: i + j + k even)
__global__ void k_mg_smooth(MgLev L, int colour, unsigned m, const unsigned *dm) {
    next_may_start();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    m = live(m, dm);
    if (t >= L.nh || !m) return;
    float c[7];
    coeffs(L, colour, t, c);
    const Nb6 n = neighbours(L.ny, L.nz, L.hx, at_of(L.nx, L.ny, L.hx, colour, t), t);
    wait_for_previous();
    if (c[0] == 0.0f) return;
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if ((m >> q) & 1u)
            split(L.x, L, q, colour)[t] =
                (split(L.b, L, q, colour)[t] - nb_sum(c, n, split(L.x, L, q, 1 - colour))) / c[0];
}

// level 0's last half-sweep (red): every cell's x to w in cell order (0 where the
// diagonal is: such a cell of the matrix is outside the mesh to the cycle)
template <class T>
__global__ void k_mg_last(MgLev L, int colour, unsigned m, const int *__restrict__ cellAt, int N, T *__restrict__ w,
                          const unsigned *dm) {
    next_may_start();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    m = live(m, dm);
    if (t >= L.nh || !m) return;
    const At a = at_of(L.nx, L.ny, L.hx, colour, t);
    const int b0 = 2 * a.ii + L.nx * (a.j + L.ny * a.k);
    const int c0 = cellAt[b0], c1 = 2 * a.ii + 1 < L.nx ? cellAt[b0 + 1] : -1;
    const int mine = a.o ? c1 : c0, other = a.o ? c0 : c1;
    float c[7];
    coeffs(L, colour, t, c);
    const Nb6 n = neighbours(L.ny, L.nz, L.hx, a, t);
    wait_for_previous();
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if ((m >> q) & 1u) {
            const float *x = split(L.x, L, q, 1 - colour);
            if (mine >= 0)
                w[(size_t)q * N + mine] = c[0] != 0.0f ? (T)((split(L.b, L, q, colour)[t] - nb_sum(c, n, x)) / c[0]) : T(0);
            if (other >= 0) w[(size_t)q * N + other] = (T)x[t];
        }
}

// the first black half-sweep after the coarse correction: the red values with
// the correction, x + kOver x_coarse(aggregate), formed as they are read
__global__ void k_mg_correct(MgLev F, MgLev C, unsigned m, const unsigned *dm) {
    next_may_start();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    m = live(m, dm);
    if (t >= F.nh || !m) return;
    float c[7];
    coeffs(F, 1, t, c);
    const At a = at_of(F.nx, F.ny, F.hx, 1, t);
    const Nb6 n = neighbours(F.ny, F.nz, F.hx, a, t);
    int B[6];   // the neighbours' aggregates: colour << 30 | entry
    {
        const int sx = F.nx != C.nx, sy = F.ny != C.ny, sz = F.nz != C.nz, i = 2 * a.ii + a.o;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            // (a neighbour outside the box has a zero coupling: any aggregate serves)
            const int I = min(max(i + (q == 0 ? -1 : q == 1 ? 1 : 0), 0), F.nx - 1) >> sx;
            const int J = min(max(a.j + (q == 2 ? -1 : q == 3 ? 1 : 0), 0), F.ny - 1) >> sy;
            const int K = min(max(a.k + (q == 4 ? -1 : q == 5 ? 1 : 0), 0), F.nz - 1) >> sz;
            B[q] = ((I + J + K) & 1) << 30 | ((K * C.ny + J) * C.hx + (I >> 1));
        }
    }
    wait_for_previous();
    if (c[0] == 0.0f) return;
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if ((m >> q) & 1u) {
            const float *x = split(F.x, F, q, 0), *xc = split(C.x, C, q, 0);
            float s = 0.0f;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const float v = __fmaf_rn(kOver, xc[(B[k] >> 30) * C.ns + (B[k] & 0x3fffffff)], x[n.i[k]]);
                s = __fmaf_rn(c[k + 1], v, s);
            }
            split(F.x, F, q, 1)[t] = (split(F.b, F, q, 1)[t] - s) / c[0];
        }
}

// the residual b - A x of each aggregate's cells, summed into the coarse
// right-hand side, and the coarse level's first red half-sweep from x = 0
__global__ void k_mg_restrict(MgLev F, MgLev C, unsigned m, const unsigned *dm) {
    next_may_start();
    const int B = blockIdx.x * blockDim.x + threadIdx.x;
    m = live(m, dm);
    if (B >= C.n || !m) return;
    int I, J, K;
    box_ijk(C, B, I, J, K);
    const int fx = F.nx == C.nx ? 1 : 2, fy = F.ny == C.ny ? 1 : 2, fz = F.nz == C.nz ? 1 : 2;
    const int colour = (I + J + K) & 1, T = (K * C.ny + J) * C.hx + (I >> 1);
    const float d = C.co[colour * C.ns + T];
    wait_for_previous();
    float s[3] = {0.0f, 0.0f, 0.0f};
    for (int dk = 0; dk < fz; ++dk)
        for (int dj = 0; dj < fy; ++dj)
            for (int di = 0; di < fx; ++di) {
                const int i = I * fx + di, j = J * fy + dj, k = K * fz + dk;
                if (i >= F.nx || j >= F.ny || k >= F.nz) continue;
                const int fc = (i + j + k) & 1, t = (k * F.ny + j) * F.hx + (i >> 1);
                float c[7];
                coeffs(F, fc, t, c);
                if (c[0] == 0.0f) continue;
                const At a{i >> 1, j, k, i & 1};
                const Nb6 n = neighbours(F.ny, F.nz, F.hx, a, t);
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    if ((m >> q) & 1u)
                        s[q] += __fmaf_rn(-c[0], split(F.x, F, q, fc)[t], split(F.b, F, q, fc)[t]) -
                                nb_sum(c, n, split(F.x, F, q, 1 - fc));
            }
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if ((m >> q) & 1u) {
            split(C.b, C, q, colour)[T] = s[q];
            if (colour == 0) split(C.x, C, q, 0)[T] = d != 0.0f ? s[q] / d : 0.0f;
        }
}

// The small levels' part of the V-cycle in one CTA: from the right-hand side
// restricted onto level `first` (and the red half-sweep of it) down to the
// coarsest level and back up to the corrected, post-smoothed x of level `first`,
// the arithmetic of the per-level passes with a barrier between them, so that
// those levels cost no launches.
//
// What bounds it: the chain of passes (13 a level, 32 on the coarsest one), each
// the latency of its loads, six products, a division and a barrier, and the
// instructions of one SM.  So everything lies in shared memory, the vectors with a
// margin of zeros as wide as a plane either side, so that a neighbour is at a
// fixed distance without a test (its coupling is zero where there is none); a
// cell's place in its pair (o) comes from a table instead of divisions; the
// coarsest level's threads hold their cells' coefficients in registers, and only
// as many warps as have cells take part there.
struct MgTail {
    MgLev lev[kMaxLevels];
    int first, n;        // levels first .. n - 1
};

// a tail level as the CTA holds it: co [7][2 colours][st], x [components][2][sv]
// (behind its first margin), b [components][2][st], o [nh] of colour 0
struct TailLev {
    int nx, ny, nz, hx, nh, n, dy, dz, st, sv;
    float *co, *x, *b;
    unsigned char *o;
};
__host__ __device__ __forceinline__ int up4(int n) { return (n + 3) & ~3; }
// the distances to the y and z neighbours (0 where there is one cell), the margin
// and the floats of a level with nq components
__host__ __device__ __forceinline__ int tail_dy(const MgLev &L) { return L.ny > 1 ? L.hx : 0; }
__host__ __device__ __forceinline__ int tail_dz(const MgLev &L) { return L.nz > 1 ? L.hx * L.ny : 0; }
__host__ __device__ __forceinline__ int tail_margin(const MgLev &L) { return up4((tail_dz(L) > tail_dy(L) ? tail_dz(L) : tail_dy(L)) + 1); }
__host__ __device__ __forceinline__ int tail_floats(const MgLev &L, int nq) {
    const int st = up4(L.nh);
    return 2 * 7 * st + 2 * nq * (st + 2 * tail_margin(L)) + 2 * nq * st + up4((L.nh + 3) / 4);
}

// threads of the CTA by components, as many as the registers allow
constexpr int tail_threads(int nq) { return nq == 1 ? 896 : nq == 2 ? 640 : 512; }

__device__ __forceinline__ void copy16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ float tail_sum(const float (&c)[7], const float *x, int t, int o, int dy, int dz) {
    float s = __fmaf_rn(c[1], x[t - 1 + o], 0.0f);
    s = __fmaf_rn(c[2], x[t + o], s);
    s = __fmaf_rn(c[3], x[t - dy], s);
    s = __fmaf_rn(c[4], x[t + dy], s);
    s = __fmaf_rn(c[5], x[t - dz], s);
    return __fmaf_rn(c[6], x[t + dz], s);
}

// a colour's half-sweep
template <int NQ>
__device__ __forceinline__ void tail_smooth(const TailLev &L, int colour) {
    const int nt = blockDim.x;
    const int nh = L.nh, dy = L.dy, dz = L.dz, st = L.st, sv = L.sv;
    const float *co = L.co + colour * st, *xo = L.x + (1 - colour) * sv, *b = L.b + colour * st;
    float *x = L.x + colour * sv;
    const unsigned char *ot = L.o;
    for (int t = threadIdx.x; t < nh; t += nt) {
        float c[7];
#pragma unroll
        for (int k = 0; k < 7; ++k) c[k] = co[2 * k * st + t];
        const int o = ot[t] ^ colour;
        if (c[0] != 0.0f)
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                x[2 * q * sv + t] = (b[2 * q * st + t] - tail_sum(c, xo + 2 * q * sv, t, o, dy, dz)) / c[0];
    }
    __syncthreads();
}

// NQ: the components of the mask
template <int NQ>
__global__ void __launch_bounds__(tail_threads(NQ), 1) k_mg_tail(MgTail T, int sweeps, unsigned m,
                                                            const unsigned *dm) {
    next_may_start();
    if (!live(m, dm)) return;
    const int nt = blockDim.x;
    extern __shared__ __align__(16) float sh[];
    __shared__ TailLev lev[kMaxLevels];
    int comp[NQ];
    for (int q = 0, k = 0; q < 3; ++q)
        if ((m >> q) & 1u) comp[k++] = q;
    if (threadIdx.x == 0) {
        float *p = sh;
        for (int l = T.first; l < T.n; ++l) {
            const MgLev &G = T.lev[l];
            TailLev &L = lev[l];
            L.nx = G.nx; L.ny = G.ny; L.nz = G.nz; L.hx = G.hx; L.nh = G.nh; L.n = G.n;
            L.dy = tail_dy(G);
            L.dz = tail_dz(G);
            const int g = tail_margin(G);
            L.st = up4(G.nh);
            L.sv = L.st + 2 * g;
            L.co = p;
            L.x = L.co + 2 * 7 * L.st + g;
            L.b = L.x - g + 2 * NQ * L.sv;
            L.o = reinterpret_cast<unsigned char *>(L.b + 2 * NQ * L.st);
            p += tail_floats(G, NQ);
        }
    }
    __syncthreads();
    for (int l = T.first; l < T.n; ++l) {
        const float *gco = T.lev[l].co;
        const size_t ns = T.lev[l].ns;
        const TailLev L = lev[l];
        const int quads = L.st / 4;
        for (int q = threadIdx.x; q < 14 * quads; q += nt) {
            const int a = q / quads, t = 4 * (q - a * quads);
            copy16(L.co + a * L.st + t, gco + a * ns + t);
        }
        float *x0 = L.x - (L.sv - L.st) / 2;
        for (int q = threadIdx.x; q < 2 * NQ * L.sv; q += nt) x0[q] = 0.0f;
        for (int t = threadIdx.x; t < L.nh; t += nt) {
            const int row = t / L.hx;
            L.o[t] = (unsigned char)((row % L.ny + row / L.ny) & 1);
        }
    }
    __syncthreads();
    wait_for_previous();
    {   // level first's right-hand side and the red half of its x
        const MgLev &G = T.lev[T.first];
        const TailLev L = lev[T.first];
        for (int t = 4 * threadIdx.x; t < L.st; t += 4 * nt)
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const float *gb = G.b + 2 * comp[q] * G.ns + t;
                copy16(L.b + 2 * q * L.st + t, gb);
                copy16(L.b + (2 * q + 1) * L.st + t, gb + G.ns);
                copy16(L.x + 2 * q * L.sv + t, G.x + 2 * comp[q] * G.ns + t);
            }
        copies_done();
    }
    __syncthreads();
    for (int l = T.first; l + 1 < T.n; ++l) {
        for (int nu = 0; nu < kNu; ++nu) {
            if (nu > 0) tail_smooth<NQ>(lev[l], 0);
            tail_smooth<NQ>(lev[l], 1);
        }
        // restriction, and the coarse level's first red half-sweep
        const TailLev F = lev[l], C = lev[l + 1];
        const int fx = F.nx == C.nx ? 1 : 2, fy = F.ny == C.ny ? 1 : 2, fz = F.nz == C.nz ? 1 : 2;
        for (int B = threadIdx.x; B < C.n; B += nt) {
            const int I = B % C.nx, r = B / C.nx, J = r % C.ny, K = r / C.ny;
            float s[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q) s[q] = 0.0f;
#pragma unroll
            for (int ch = 0; ch < 8; ++ch) {
                const int di = ch & 1, dj = ch >> 1 & 1, dk = ch >> 2;
                const int i = I * fx + di, j = J * fy + dj, k = K * fz + dk;
                if (di < fx && dj < fy && dk < fz && i < F.nx && j < F.ny && k < F.nz) {
                    const int fc = (i + j + k) & 1, t = (k * F.ny + j) * F.hx + (i >> 1);
                    float c[7];
#pragma unroll
                    for (int q = 0; q < 7; ++q) c[q] = F.co[(2 * q + fc) * F.st + t];
                    if (c[0] != 0.0f)
#pragma unroll
                        for (int q = 0; q < NQ; ++q)
                            s[q] += __fmaf_rn(-c[0], F.x[(2 * q + fc) * F.sv + t], F.b[(2 * q + fc) * F.st + t]) -
                                    tail_sum(c, F.x + (2 * q + 1 - fc) * F.sv, t, i & 1, F.dy, F.dz);
                }
            }
            const int colour = (I + J + K) & 1, t = (K * C.ny + J) * C.hx + (I >> 1);
            const float d = C.co[colour * C.st + t];
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                C.b[(2 * q + colour) * C.st + t] = s[q];
                if (colour == 0) C.x[2 * q * C.sv + t] = d != 0.0f ? s[q] / d : 0.0f;
            }
        }
        __syncthreads();
    }
    {   // the coarsest level: `sweeps` symmetric sweeps (red, black, black, red)
        // from x = 0, the first red half done.  A second half-sweep of a colour
        // in a row changes nothing (it reads the other colour and b alone), so
        // black, red a sweep are the same sweeps.
        const TailLev L = lev[T.n - 1];
        if (L.nh <= nt) {
            const int part = ((L.nh + 31) >> 5) * 32, t = threadIdx.x;
            if (t < part) {
                // this thread's red and black cell, their coefficients in registers
                float c[2][7], rb[2][NQ];
                const int o = t < L.nh ? L.o[t] : 0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int k = 0; k < 7; ++k) c[h][k] = t < L.nh ? L.co[(2 * k + h) * L.st + t] : 0.0f;
#pragma unroll
                    for (int q = 0; q < NQ; ++q) rb[h][q] = t < L.nh ? L.b[(2 * q + h) * L.st + t] : 0.0f;
                }
                for (int s = 0; s < sweeps; ++s)
#pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        const int h = 1 - g;
                        if (c[h][0] != 0.0f)
#pragma unroll
                            for (int q = 0; q < NQ; ++q)
                                L.x[(2 * q + h) * L.sv + t] =
                                    (rb[h][q] - tail_sum(c[h], L.x + (2 * q + 1 - h) * L.sv, t, o ^ h, L.dy, L.dz)) / c[h][0];
                        asm volatile("bar.sync 1, %0;" ::"r"(part) : "memory");
                    }
            }
            __syncthreads();
        } else {
            for (int s = 0; s < sweeps; ++s) {
                tail_smooth<NQ>(lev[T.n - 1], 1);
                tail_smooth<NQ>(lev[T.n - 1], 0);
            }
        }
    }
    for (int l = T.n - 2; l >= T.first; --l) {
        {   // the coarse correction of the red cells (the black ones' x is
            // overwritten next, unread)
            const TailLev F = lev[l], C = lev[l + 1];
            const int sx = F.nx != C.nx, sy = F.ny != C.ny, sz = F.nz != C.nz;
            for (int t = threadIdx.x; t < F.nh; t += nt) {
                const int row = t / F.hx, j = row % F.ny, k = row / F.ny, i = 2 * (t - row * F.hx) + ((j + k) & 1);
                if (F.co[t] == 0.0f) continue;
                const int I = i >> sx, J = j >> sy, K = k >> sz;
                const int B = ((I + J + K) & 1) * C.sv + (K * C.ny + J) * C.hx + (I >> 1);
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    F.x[2 * q * F.sv + t] = __fmaf_rn(kOver, C.x[2 * q * C.sv + B], F.x[2 * q * F.sv + t]);
            }
            __syncthreads();
        }
        for (int nu = 0; nu < kNu; ++nu) {
            tail_smooth<NQ>(lev[l], 1);
            tail_smooth<NQ>(lev[l], 0);
        }
    }
    {   // level first's x, for the level above
        const MgLev &G = T.lev[T.first];
        const TailLev L = lev[T.first];
        for (int t = 4 * threadIdx.x; t < L.st; t += 4 * nt)
#pragma unroll
            for (int q = 0; q < NQ; ++q)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    *reinterpret_cast<float4 *>(G.x + (2 * comp[q] + h) * G.ns + t) =
                        *reinterpret_cast<const float4 *>(L.x + (2 * q + h) * L.sv + t);
    }
}

std::vector<MgLev> levels(rt_ctx *ctx, bool sym) {
    StructMesh &s = ctx->mesh.sm;
    std::vector<MgLev> out;
    float *p = s.mgData.p;
    for (const auto &d : s.mgDims) {
        MgLev L{};
        L.nx = d[0];
        L.ny = d[1];
        L.nz = d[2];
        L.n = d[0] * d[1] * d[2];
        L.hx = (d[0] + 1) / 2;
        L.nh = L.hx * d[1] * d[2];
        L.np = ((size_t)L.n + 31) / 32 * 32;
        L.ns = ((size_t)L.nh + 31) / 32 * 32;
        float *q = p;
        L.dg = q;
        L.xl = q + L.np;
        L.yl = q + 2 * L.np;
        L.zl = q + 3 * L.np;
        L.xu = sym ? L.xl : q + 4 * L.np;
        L.yu = sym ? L.yl : q + 5 * L.np;
        L.zu = sym ? L.zl : q + 6 * L.np;
        q += kBoxArrays * L.np;
        L.co = q;
        L.x = L.co + 2 * 7 * L.ns;
        L.b = L.x + 2 * 3 * L.ns;
        p = q + kSplitArrays * L.ns;
        out.push_back(L);
    }
    return out;
}

}  // namespace

bool mg_available(rt_ctx *ctx) {
    const DevMesh &m = ctx->mesh;
    return m.sm.on && !m.hasCoupled && m.sm.boxOf.p != nullptr;
}

void mg_prepare(rt_ctx *ctx, const double *diag, const double *upper, const double *lower, bool sym) {
    StructMesh &s = ctx->mesh.sm;
    const int N = ctx->mesh.N;
    if (s.mgDims.empty()) {   // the hierarchy's boxes, once per mesh
        int nx = s.nx, ny = s.ny, nz = s.nz;
        size_t total = 0;
        for (;;) {
            s.mgDims.push_back({nx, ny, nz});
            total += kBoxArrays * (((size_t)nx * ny * nz + 31) / 32 * 32) +
                     kSplitArrays * (((size_t)(nx + 1) / 2 * ny * nz + 31) / 32 * 32);
            if ((long long)nx * ny * nz <= kCoarse || (nx == 1 && ny == 1 && nz == 1)) break;
            RT_REQUIRE((int)s.mgDims.size() < kMaxLevels, RT_EINVAL, "multigrid: too many levels");
            nx = (nx + 1) / 2;
            ny = (ny + 1) / 2;
            nz = (nz + 1) / 2;
        }
        s.mgData.alloc(total);
        s.mgData.zero(ctx->stream);   // (x stays zero outside the mesh)
    }
    std::vector<MgLev> L = levels(ctx, sym);
    RT_CUDA(cudaMemsetAsync(L[0].dg, 0, sizeof(float) * L[0].np * 7, ctx->stream));
    k_mg_fine<<<nblocks(N), RT_BLOCK, 0, ctx->stream>>>(N, s.boxOf.p, s.faceLo.p, diag, upper, lower, L[0],
                                                       sym ? 1 : 0);
    for (size_t l = 1; l < L.size(); ++l)
        k_mg_coarsen<<<nblocks(L[l].n), RT_BLOCK, 0, ctx->stream>>>(L[l - 1], L[l], sym ? 1 : 0);
    for (const MgLev &l : L) k_mg_split<<<nblocks(2 * l.nh), RT_BLOCK, 0, ctx->stream>>>(l);
    RT_CHECK_LAUNCH();
    launch_count(ctx, 2 * (int)L.size());
}

namespace {

void launch_tail(const std::vector<MgLev> &L, int first, unsigned m, const unsigned *dm, cudaStream_t st) {
    MgTail tail{};
    for (size_t l = 0; l < L.size(); ++l) tail.lev[l] = L[l];
    tail.first = first;
    tail.n = (int)L.size();
    const int nq = __builtin_popcount(m & 7u);
    size_t bytes = 0;
    for (size_t l = first; l < L.size(); ++l) bytes += tail_floats(L[l], nq) * sizeof(float);
    RT_REQUIRE(bytes <= kTailSmem, RT_EINVAL, "multigrid: the coarsest level does not fit one CTA");
    auto k = nq == 1 ? k_mg_tail<1> : nq == 2 ? k_mg_tail<2> : k_mg_tail<3>;
    RT_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailSmem));
    const int threads = std::min(tail_threads(nq), std::max(128, (L[first].nh + 31) / 32 * 32));
    launch_next(k, 1, threads, bytes, st, tail, kCoarseSweeps, m, dm);
}

// one V-cycle's launches on the stream; the number of kernels
template <class T>
int enqueue_vcycle(rt_ctx *ctx, const std::vector<MgLev> &L, unsigned m, const T *r, T *w, const unsigned *dm) {
    StructMesh &s = ctx->mesh.sm;
    cudaStream_t st = ctx->stream;
    const int N = ctx->mesh.N;
    const int nL = (int)L.size();
    int launches = 0;
    auto blocks = [](int n) { return nblocks(n, kPassBlock); };
    auto smooth = [&](const MgLev &l, int colour) {
        launch_next(k_mg_smooth, blocks(l.nh), kPassBlock, 0, st, l, colour, m, dm);
        ++launches;
    };
    // the levels that run in one CTA: the coarsest and those above it that are
    // small and fit (not level 0 above others: its first and last passes read r
    // and write w in cell order)
    int tf = nL - 1;
    size_t floats = tail_floats(L[tf], __builtin_popcount(m & 7u));
    while (tf > 1 && L[tf - 1].n <= kTailCells) {
        floats += tail_floats(L[tf - 1], __builtin_popcount(m & 7u));
        if (floats * sizeof(float) > kTailSmem) break;
        --tf;
    }
    k_mg_first<T><<<blocks(L[0].nh), kPassBlock, 0, st>>>(L[0], s.cellAt.p, N, m, r, dm);
    ++launches;
    // down: pre-smoothing (kNu sweeps, red then black; the first red half is
    // done) and restriction
    for (int l = 0; l < tf; ++l) {
        for (int nu = 0; nu < kNu; ++nu) {
            if (nu > 0) smooth(L[l], 0);
            smooth(L[l], 1);
        }
        launch_next(k_mg_restrict, blocks(L[l + 1].n), kPassBlock, 0, st, L[l], L[l + 1], m, dm);
        ++launches;
    }
    launch_tail(L, tf, m, dm, st);
    ++launches;
    if (nL == 1) {
        // a mesh no larger than the coarsest level: its x to w.  The sweeps ended on
        // red, and the same half-sweep again changes nothing; one more on black would
        // make the cycle unsymmetric, which PCG pays for (16 x 16 cells 18 iterations
        // against 12, 128 x 4 91 against 71)
        launch_next(k_mg_last<T>, blocks(L[0].nh), kPassBlock, 0, st, L[0], 0, m, (const int *)s.cellAt.p, N, w, dm);
        RT_CHECK_LAUNCH();
        return launches + 1;
    }
    // up: the coarse correction and post-smoothing (black, red); level 0's last
    // half-sweep writes w
    for (int l = tf - 1; l >= 0; --l)
        for (int nu = 0; nu < kNu; ++nu) {
            if (nu == 0) {
                launch_next(k_mg_correct, blocks(L[l].nh), kPassBlock, 0, st, L[l], L[l + 1], m, dm);
                ++launches;
            } else {
                smooth(L[l], 1);
            }
            if (l == 0 && nu == kNu - 1) {
                launch_next(k_mg_last<T>, blocks(L[l].nh), kPassBlock, 0, st, L[l], 0, m, (const int *)s.cellAt.p, N, w, dm);
                ++launches;
            } else {
                smooth(L[l], 0);
            }
        }
    RT_CHECK_LAUNCH();
    return launches;
}

// The V-cycle's launches are captured once into a CUDA graph (per mesh,
// matrix kind and r, w, dm buffers and components: a Krylov loop passes the
// same few every iteration) and the graph is launched per application: most
// of the levels are small, and their launches, not their data, set the
// V-cycle's time.
template <class T>
void apply(rt_ctx *ctx, bool sym, unsigned m, const T *r, T *w, const unsigned *dm) {
    StructMesh &s = ctx->mesh.sm;
    MgGraph *gr = nullptr;
    for (MgGraph &g : s.mgGraph)
        if (g.exec && g.r == r && g.w == w && g.dm == dm && g.mask == m && g.sym == sym) gr = &g;
    if (!gr) {
        gr = &s.mgGraph[s.mgNext];
        s.mgNext = (s.mgNext + 1) % kMgGraphs;
        gr->reset();
        std::vector<MgLev> L = levels(ctx, sym);
        cudaGraph_t g = nullptr;
        RT_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        int n = 0;
        try {
            n = enqueue_vcycle<T>(ctx, L, m, r, w, dm);
        } catch (...) {
            cudaGraph_t dead = nullptr;
            cudaStreamEndCapture(ctx->stream, &dead);
            if (dead) cudaGraphDestroy(dead);
            throw;
        }
        RT_CUDA(cudaStreamEndCapture(ctx->stream, &g));
        cudaGraphExec_t exec = nullptr;
        const cudaError_t e = cudaGraphInstantiate(&exec, g, 0);
        cudaGraphDestroy(g);
        RT_CUDA(e);
        gr->exec = exec;
        gr->r = r;
        gr->w = w;
        gr->dm = dm;
        gr->mask = m;
        gr->sym = sym;
        gr->launches = n;
    }
    RT_CUDA(cudaGraphLaunch(gr->exec, ctx->stream));
    launch_count(ctx, gr->launches);
}

}  // namespace

void mg_apply(rt_ctx *ctx, const double *r, double *w, const unsigned *dm) {
    apply<double>(ctx, true, 1u, r, w, dm);
}

void mg_apply32(rt_ctx *ctx, unsigned mask, const float *r, float *w, const unsigned *dm) {
    apply<float>(ctx, false, mask, r, w, dm);
}

}  // namespace rt
