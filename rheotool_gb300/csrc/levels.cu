// levels.cu — DIC / DILU factorisation and sweeps on any mesh, level by level
// inside one kernel.
//
// The cells of a level (1 + the highest level of a cell's lower neighbours)
// depend only on cells of lower levels.  The cells are renumbered by level, so
// that a level is a contiguous range of positions; a position keeps the
// positions of its lower and upper neighbours in face order and, per matrix,
// the premultiplied coefficients rD a.  An application of the preconditioner is
// one launch: a CTA (or a cluster of eight) a component walks the levels up and
// down with a barrier between them, in the sequential sweep's order of
// operations in each cell.
//
// What bounds it: a mesh has a few hundred levels of a few dozen to a few
// thousand cells, so the time is that of the dependent chain of levels.  One
// launch a level costs a launch, about 5 us, on either sweep; here a level costs
// the barrier, the loads of the neighbours' values and the products: with the
// values in shared memory about 0.2 us.  The coefficients of a thread's first
// cells of the next levels are loaded ahead of them.
#include <algorithm>

#include "real_ops.cuh"
#include "rt_internal.h"
#include "sweep.h"

namespace rt {

namespace {

// A cell's first NP neighbours (3, or 2 where no cell has more: FP64 products of
// an absent third one cost a level a sixth of its time) are loaded kDeep levels
// ahead, the others when they are needed.  Measured on 2-D contraction of 7,200 cells,
// an application: FP64 113 us with NP = 2, 140 with 3; FP32 96 us with two levels
// ahead, 115 with one, 95 with four (FP64 153 with four).
constexpr int kDeep = 2;
constexpr int kMaxThreads = 1024;
constexpr size_t kMaxSmem = 220 * 1024;

// the levels' positions (built on first use, kept with the mesh)
struct LevelView {
    int N, nl, nLo, nUp, width;                  // cells, levels, neighbours a cell at most, cells a level at most
    const int *__restrict__ start;               // nl + 1
    const int *__restrict__ cell;                // N: the cell of each position
    const int *__restrict__ lo, *__restrict__ loFace;   // [slot][position]: face order, -1 ends a row
    const int *__restrict__ up, *__restrict__ upFace;   // faces descending
};

__global__ void k_level_pos(int N, const int *__restrict__ cell, int *__restrict__ posOf) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < N) posOf[cell[p]] = p;
}

__global__ void k_level_maps(int N, int nLo, int nUp, const int *__restrict__ cell, const int *__restrict__ posOf,
                             const int *__restrict__ plNbr, const int *__restrict__ plFace,
                             const int *__restrict__ puNbr, const int *__restrict__ puFace, int *__restrict__ lo,
                             int *__restrict__ loFace, int *__restrict__ up, int *__restrict__ upFace) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= N) return;
    const int c = cell[p];
    for (int s = 0; s < nLo; ++s) {
        const int nb = plNbr[(size_t)s * N + c];
        lo[(size_t)s * N + p] = nb >= 0 ? posOf[nb] : -1;
        loFace[(size_t)s * N + p] = plFace[(size_t)s * N + c];
    }
    int n = 0;
    while (n < nUp && puNbr[(size_t)n * N + c] >= 0) ++n;
    for (int s = 0; s < nUp; ++s) {
        const int q = n - 1 - s;
        up[(size_t)s * N + p] = q >= 0 ? posOf[puNbr[(size_t)q * N + c]] : -1;
        upFace[(size_t)s * N + p] = q >= 0 ? puFace[(size_t)q * N + c] : -1;
    }
}

LevelView level_view(rt_ctx *ctx) {
    DevMesh &m = ctx->mesh;
    LevelMesh &l = m.lev;
    const size_t N = m.N, nLo = std::max(m.pnLo, 1), nUp = std::max(m.pnUp, 1);
    if (!l.ready) {
        l.maps.alloc((2 * nLo + 2 * nUp) * N);
        l.start.upload(m.levelStartH.data(), m.levelStartH.size(), ctx->stream);
        DBuf<int> pos;
        pos.alloc(N);
        int *p = l.maps.p;
        k_level_pos<<<nblocks(N), RT_BLOCK, 0, ctx->stream>>>((int)N, m.levelCells.p, pos.p);
        k_level_maps<<<nblocks(N), RT_BLOCK, 0, ctx->stream>>>((int)N, m.pnLo, m.pnUp, m.levelCells.p, pos.p, m.plNbr.p,
                                                               m.plFace.p, m.puNbr.p, m.puFace.p, p, p + nLo * N,
                                                               p + 2 * nLo * N, p + (2 * nLo + nUp) * N);
        RT_CHECK_LAUNCH();
        launch_count(ctx, 2);
        RT_CUDA(cudaStreamSynchronize(ctx->stream));   // (pos, levelStartH)
        l.width = 0;
        for (int i = 0; i < m.nLevels; ++i) l.width = std::max(l.width, m.levelStartH[i + 1] - m.levelStartH[i]);
        l.ready = true;
    }
    int *p = l.maps.p;
    return LevelView{m.N, m.nLevels, m.pnLo, m.pnUp, l.width, l.start.p, m.levelCells.p, p, p + nLo * N,
                     p + 2 * nLo * N, p + (2 * nLo + nUp) * N};
}

// the premultiplied coefficients of one matrix by position: rd, lo[slot], up[slot]
template <class Real>
struct LevelCoef {
    Real *rd, *lo, *up;
};

template <class Real>
LevelCoef<Real> coef_view(rt_ctx *ctx, DBuf<Real> &buf) {
    const DevMesh &m = ctx->mesh;
    const size_t N = m.N, need = (1 + (size_t)m.pnLo + m.pnUp) * N;
    if (buf.n != need) buf.alloc(need);
    return LevelCoef<Real>{buf.p, buf.p + N, buf.p + (1 + (size_t)m.pnLo) * N};
}

// rD: the reciprocal diagonal in cell order
template <class Real>
__global__ void k_level_coef(LevelView v, LevelCoef<Real> a, const Real *__restrict__ rD, const Real *__restrict__ lower,
                             const Real *__restrict__ upper) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= v.N) return;
    const Real rd = rD[v.cell[p]];
    a.rd[p] = rd;
    for (int s = 0; s < v.nLo; ++s) {
        const int f = v.loFace[(size_t)s * v.N + p];
        a.lo[(size_t)s * v.N + p] = f >= 0 ? r_mul(rd, lower[f]) : Real(0);
    }
    for (int s = 0; s < v.nUp; ++s) {
        const int f = v.upFace[(size_t)s * v.N + p];
        a.up[(size_t)s * v.N + p] = f >= 0 ? r_mul(rd, upper[f]) : Real(0);
    }
}

// a barrier of the threads that walk the levels: `n` threads of this CTA, or
// every thread of the cluster
template <int CS>
__device__ __forceinline__ void level_barrier(int n) {
    if (CS > 1) asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
    else asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
}
// values other CTAs of the cluster wrote are read from L2
template <int CS, class T>
__device__ __forceinline__ T value(const T *p) {
    return CS > 1 ? __ldcg(p) : *p;
}

// one triangular sweep over the levels, x in place: x -= sum coef x(neighbour)
template <class Real, int CS, int NP, bool UP>
__device__ void level_sweep(const LevelView &v, const int *start, Real *x, const int *__restrict__ nbr,
                            const Real *__restrict__ coef, int nSlots, int tid, int nt) {
    // the thread's first cells of the next kDeep levels
    int d[kDeep][NP];
    Real c[kDeep][NP];
    const int first = UP ? v.nl - 2 : 1, last = UP ? -1 : v.nl, step = UP ? -1 : 1;
    auto ahead = [&](int l, int (&dl)[NP], Real (&cl)[NP]) {
        const bool level = UP ? l > last : l < last;
        const int p = level ? start[l] + tid : 0;
        const bool in = level && p < start[l + 1];
#pragma unroll
        for (int s = 0; s < NP; ++s) {
            dl[s] = in && s < nSlots ? nbr[(size_t)s * v.N + p] : -1;
            cl[s] = in && s < nSlots ? coef[(size_t)s * v.N + p] : Real(0);
        }
    };
    if (v.nl < 2) return;
#pragma unroll
    for (int q = 0; q < kDeep; ++q) ahead(first + q * step, d[q], c[q]);
    for (int l = first; l != last; l += step) {
        const int p0 = start[l] + tid, end = start[l + 1];
        int d0[NP];
        Real c0[NP];
#pragma unroll
        for (int s = 0; s < NP; ++s) {
            d0[s] = d[0][s];
            c0[s] = c[0][s];
#pragma unroll
            for (int q = 0; q + 1 < kDeep; ++q) {
                d[q][s] = d[q + 1][s];
                c[q][s] = c[q + 1][s];
            }
        }
        ahead(l + kDeep * step, d[kDeep - 1], c[kDeep - 1]);
        if (p0 < end) {
            Real acc = value<CS>(x + p0), xn[NP];
#pragma unroll
            for (int s = 0; s < NP; ++s) xn[s] = d0[s] >= 0 ? value<CS>(x + d0[s]) : Real(0);
#pragma unroll
            for (int s = 0; s < NP; ++s)
                if (d0[s] >= 0) acc = r_fma(-c0[s], xn[s], acc);
            for (int s = NP; s < nSlots; ++s) {
                const int q = nbr[(size_t)s * v.N + p0];
                if (q < 0) break;
                acc = r_fma(-coef[(size_t)s * v.N + p0], value<CS>(x + q), acc);
            }
            x[p0] = acc;
        }
        for (int p = p0 + nt; p < end; p += nt) {
            Real acc = value<CS>(x + p);
            for (int s = 0; s < nSlots; ++s) {
                const int q = nbr[(size_t)s * v.N + p];
                if (q < 0) break;
                acc = r_fma(-coef[(size_t)s * v.N + p], value<CS>(x + q), acc);
            }
            x[p] = acc;
        }
        level_barrier<CS>(nt);
    }
}

// what lies in shared memory: the values (behind the starts), the levels' starts (all
// but a chain of some 55,000 levels; those are read where they are)
constexpr int kValuesIn = 1, kStartsIn = 2;
__device__ __forceinline__ const int *level_starts(const LevelView &v, unsigned char *smem, int inSmem) {
    if (!(inSmem & kStartsIn)) return v.start;
    int *start = reinterpret_cast<int *>(smem);
    for (int i = threadIdx.x; i <= v.nl; i += blockDim.x) start[i] = v.start[i];
    return start;   // (the caller has a barrier before it reads them)
}

// w = M^-1 r of component blockIdx.x / CS of the masked ones, forward and
// backward.  x holds the values by position: in shared memory (CS == 1 and
// they fit) or in `scratch`.
template <class Real, int CS, int NP>
__global__ void __launch_bounds__(kMaxThreads) k_level_apply(LevelView v, LevelCoef<Real> a, unsigned mask, int walkers,
                                                            int inSmem, const Real *r, Real *w, Real *scratch,
                                                            const unsigned *dmask) {
    extern __shared__ __align__(16) unsigned char smem[];
    next_may_start();
    const int *start = level_starts(v, smem, inSmem);
    wait_for_previous();
    const unsigned live = dmask ? mask & *dmask : mask;
    unsigned m = mask;
    for (int q = blockIdx.x / CS; q > 0; --q) m &= m - 1;
    const int comp = __ffs(m) - 1;
    if (!((live >> comp) & 1u)) return;   // (every CTA of the cluster alike)
    Real *x = inSmem & kValuesIn ? reinterpret_cast<Real *>(smem + ((size_t)(v.nl + 1) * 4 + 15) / 16 * 16)
                     : scratch + (size_t)comp * v.N;
    r += (size_t)comp * v.N;
    w += (size_t)comp * v.N;
    const int rank = CS > 1 ? blockIdx.x % CS : 0;
    const int all = CS * blockDim.x, tid = rank * blockDim.x + threadIdx.x;
    for (int p = tid; p < v.N; p += all) x[p] = r_mul(a.rd[p], r[v.cell[p]]);
    __syncthreads();
    if (CS > 1) level_barrier<CS>(0);
    const int nt = CS > 1 ? all : walkers;
    if (tid < nt) {
        level_sweep<Real, CS, NP, false>(v, start, x, v.lo, a.lo, v.nLo, tid, nt);
        level_sweep<Real, CS, NP, true>(v, start, x, v.up, a.up, v.nUp, tid, nt);
    }
    __syncthreads();
    for (int p = tid; p < v.N; p += all) w[v.cell[p]] = value<CS>(x + p);
}

// rD of the factorisation, by position in `x` (as in k_level_apply), then its
// reciprocal in cell order
template <int CS>
__global__ void __launch_bounds__(kMaxThreads) k_level_factor(LevelView v, int walkers, int inSmem,
                                                             const double *diag, const double *upper,
                                                             const double *lower, double *scratch, double *rD) {
    after_previous();
    extern __shared__ __align__(16) unsigned char smem[];
    const int *start = level_starts(v, smem, inSmem);
    double *x = inSmem & kValuesIn ? reinterpret_cast<double *>(smem + ((size_t)(v.nl + 1) * 4 + 15) / 16 * 16) : scratch;
    const int rank = CS > 1 ? blockIdx.x % CS : 0;
    const int all = CS * blockDim.x, tid = rank * blockDim.x + threadIdx.x;
    for (int p = tid; p < v.N; p += all) x[p] = diag[v.cell[p]];
    __syncthreads();
    if (CS > 1) level_barrier<CS>(0);
    const int nt = CS > 1 ? all : walkers;
    if (tid < nt)
        for (int l = 1; l < v.nl; ++l) {
            for (int p = start[l] + tid; p < start[l + 1]; p += nt) {
                double acc = value<CS>(x + p);
                for (int s = 0; s < v.nLo; ++s) {
                    const int q = v.lo[(size_t)s * v.N + p];
                    if (q < 0) break;
                    const int f = v.loFace[(size_t)s * v.N + p];
                    acc = __dsub_rn(acc, __ddiv_rn(__dmul_rn(upper[f], lower[f]), value<CS>(x + q)));
                }
                x[p] = acc;
            }
            level_barrier<CS>(nt);
        }
    __syncthreads();
    for (int p = tid; p < v.N; p += all) rD[v.cell[p]] = 1.0 / value<CS>(x + p);
}

struct LevelLaunch {
    int CS, threads, walkers, inSmem;
    size_t smem;
};

// One CTA a component, or a cluster of eight where the widest level takes one CTA
// more than `passes` passes of its threads: a cluster's barrier and values through
// L2 cost a level more (contraction of 38k cells, widest level 900: 253 us an
// application in one CTA, 409 in eight; 127k cells: 680 and 693; 1M cells, 4,000
// wide: 7,330 and 1,910; one launch a level took 1,690, 2,660 and 7,660).
LevelLaunch plan(const LevelView &v, size_t real, int passes) {
    LevelLaunch q{};
    const size_t starts = ((size_t)(v.nl + 1) * 4 + 15) / 16 * 16, vals = (size_t)v.N * real;
    q.CS = v.width > passes * kMaxThreads ? 8 : 1;
    q.inSmem = (q.CS == 1 && starts + vals <= kMaxSmem ? kValuesIn : 0) | (starts <= kMaxSmem ? kStartsIn : 0);
    q.smem = (q.inSmem & kStartsIn ? starts : 0) + (q.inSmem & kValuesIn ? vals : 0);
    q.threads = kMaxThreads;
    q.walkers = std::min(kMaxThreads, (v.width + 31) / 32 * 32);
    return q;
}

template <class... A>
void launch_levels(rt_ctx *ctx, void (*one)(A...), void (*eight)(A...), const LevelLaunch &q, int ncomp, A... args) {
    void (*k)(A...) = q.CS == 1 ? one : eight;
    if (q.smem > 40 * 1024)
        RT_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(q.CS * ncomp);
    cfg.blockDim = dim3(q.threads);
    cfg.dynamicSmemBytes = q.smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // (see launch_next)
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = q.CS;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = q.CS > 1 ? 2 : 1;
    RT_CUDA(cudaLaunchKernelEx(&cfg, k, args...));
    RT_CHECK_LAUNCH();
    launch_count(ctx);
}

template <class Real>
Real *scratch(rt_ctx *ctx, const LevelLaunch &q, int ncomp) {
    if (q.inSmem & kValuesIn) return nullptr;
    DBuf<double> &b = ctx->mesh.lev.scratch;
    const size_t need = ((size_t)ctx->mesh.N * ncomp * sizeof(Real) + 7) / 8;
    if (b.n < need) b.alloc(need);
    return reinterpret_cast<Real *>(b.p);
}

template <class Real>
void apply(rt_ctx *ctx, DBuf<Real> &coef, unsigned mask, const Real *r, Real *w, const unsigned *dmask) {
    if (!mask) return;
    const LevelView v = level_view(ctx);
    const LevelLaunch q = plan(v, sizeof(Real), 3);
    const bool two = std::max(v.nLo, v.nUp) <= 2;
    launch_levels(ctx, two ? k_level_apply<Real, 1, 2> : k_level_apply<Real, 1, 3>,
                  two ? k_level_apply<Real, 8, 2> : k_level_apply<Real, 8, 3>, q, __builtin_popcount(mask), v,
                  coef_view(ctx, coef), mask, q.walkers, q.inSmem, r, w, scratch<Real>(ctx, q, 32 - __builtin_clz(mask)),
                  dmask);
}

}  // namespace

void level_factor(rt_ctx *ctx, const double *diag, const double *upper, const double *lower, double *rD) {
    const LevelView v = level_view(ctx);
    const LevelLaunch q = plan(v, sizeof(double), 1);   // (a cell's divisions take a CTA's FP64 units longer)
    launch_levels(ctx, k_level_factor<1>, k_level_factor<8>, q, 1, v, q.walkers, q.inSmem, diag, upper, lower,
                  scratch<double>(ctx, q, 1), rD);
}

void level_coefs(rt_ctx *ctx, const double *rD, const double *lower, const double *upper, bool T) {
    const LevelView v = level_view(ctx);
    LevelMesh &l = ctx->mesh.lev;
    k_level_coef<double><<<nblocks(v.N), RT_BLOCK, 0, ctx->stream>>>(v, coef_view(ctx, T ? l.coefT : l.coef), rD,
                                                                    T ? upper : lower, T ? lower : upper);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
}

void level_coefs32(rt_ctx *ctx, const float *rD, const float *lower, const float *upper) {
    const LevelView v = level_view(ctx);
    k_level_coef<float><<<nblocks(v.N), RT_BLOCK, 0, ctx->stream>>>(v, coef_view(ctx, ctx->mesh.lev.coef32), rD, lower,
                                                                   upper);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
}

void level_precondition(rt_ctx *ctx, unsigned mask, const double *r, double *w, bool T, const unsigned *dmask) {
    LevelMesh &l = ctx->mesh.lev;
    apply<double>(ctx, T ? l.coefT : l.coef, mask, r, w, dmask);
}

void level_precondition32(rt_ctx *ctx, unsigned mask, const float *r, float *w, const unsigned *dmask) {
    apply<float>(ctx, ctx->mesh.lev.coef32, mask, r, w, dmask);
}

}  // namespace rt
