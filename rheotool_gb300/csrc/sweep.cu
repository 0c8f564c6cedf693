// sweep.cu — systolic triangular sweeps of DIC / DILU on structured meshes.
//
// A structured mesh is the active-cell subset of an nx x ny x nz box numbered
// lexicographically (i fastest), as blockMesh numbers a block.  Its lower
// neighbours are (i,j,k-1), (i,j-1,k), (i-1,j,k) in increasing face order, its
// upper neighbours (i+1,j,k), (i,j+1,k), (i,j,k+1).  The sequential D-ILU
// recurrences of OpenFOAM (rD, forward, backward; face-ordered accumulation)
// are evaluated here in exactly that order of operations, so the FP64 result
// equals the level-scheduled sweep bit for bit (and the sequential sweep up to
// FMA contraction).  The same kernel runs in FP32 for the mixed-precision
// solvers (coefficients rounded from the FP64 factorisation).
//
// Work decomposition: the rows (j, k) are grouped in tiles of TJ x TK = 32 (8 x
// 4, or 32 x 1 on a mesh of one plane), a tile a warp and a row a lane, and WJ
// x WK neighbouring tiles in a CTA.  At step t the lane of row (j, k) of its
// tile updates cell i = t - kSkewJ j - kSkewK k.  The i-1 value is the lane's own
// last result; the j-1 and k-1 values are results that other lanes formed, read
// from a ring of the last steps' results of all the CTA's tiles in shared
// memory; those of the tiles of other CTAs (the ghosts) lie in the same ring.  So
// a lane reads its two neighbours at addresses fixed but for the step, and a
// step is two reads, three products and one write, without a branch.
//
// What bounds it: latency.  Measured on GB300: a dependent FP64 fused
// multiply-add takes a warp 64 cycles and an independent one 48 (one FP64 unit
// a quarter of an SM, whatever the lanes in use), an FP32 one 4; an FP64 result
// reaches shared memory 105 cycles after its product; a value takes 35 through
// shared memory and 480 to 860 through L2 to another SM.  So an FP64 step cannot
// take less than about 245 cycles and an FP32 one 45; the longest chain has nx +
// kSkewJ ny + kSkewK nz steps.  So four tiles of a CTA (one a quarter
// of the SM) hand over in shared memory, only every second tile boundary
// goes through L2, and all else is kept off the tiles' warps: other warps of
// the CTA fetch the ghosts, hand results to the next CTAs, stage coefficients
// and write results out.  (A skew of two in k would take the k product off a
// step's chain, but a warp issues its FP64 products in order: a step was no shorter,
// and there were nz more of them.  The rD recurrence, three quotients a step, hands
// each value on with its reciprocal, which leaves five products of a quotient: 616 us
// for 1M cells against 1370 with three divisions, 287 against 667 for 127k.)
//
// A value handed to another CTA is its own flag: the hand-off words hold the
// pattern of all ones until the producer writes the value (a result with that
// pattern, a NaN, is written as another NaN), and the consumer puts the
// pattern back once it has read the word.  So a consumer waits on the data
// itself, one L2 round trip after the store; no fence, tag or release/acquire
// pair sits on the dependency chain.  Groups of tiles are taken in dependency
// order from an atomic counter, so a CTA only waits on CTAs already running: no
// deadlock.  Every wait is bounded; a timeout sets an error flag, every other
// wait gives up on seeing it, and the host reports RT_ETIMEOUT and clears the
// hand-off words.
//
// Per-entry data live in a "skewed" layout of (tile, step, lane) in which one
// lane's two consecutive steps are adjacent (a pair), so a lane reads and
// writes its coefficients and results as 16-byte vectors without bank
// conflicts, and a chunk of P steps of one array is one contiguous block,
// staged by one bulk copy NB chunks ahead.  The backward sweep walks the
// same layout in reverse (lanes mirrored).
#include <algorithm>

#include "real_ops.cuh"
#include "rt_internal.h"
#include "sweep.h"

namespace rt {

typedef unsigned long long u64;

// ---- hand-off words ---------------------------------------------------------
template <class Real> struct Word;
template <> struct Word<double> {
    typedef u64 T;
    static __device__ __forceinline__ T of(double v) { return (T)__double_as_longlong(v); }
    static __device__ __forceinline__ double value(T w) { return __longlong_as_double((long long)w); }
    static constexpr T kOtherNaN = 0x7ff8000000000000ull;
};
template <> struct Word<float> {
    typedef unsigned T;
    static __device__ __forceinline__ T of(float v) { return __float_as_uint(v); }
    static __device__ __forceinline__ float value(T w) { return __uint_as_float(w); }
    static constexpr T kOtherNaN = 0x7fc00000u;
};
__device__ __forceinline__ u64 ld_word(const u64 *p) {
    u64 v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned ld_word(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void st_word(u64 *p, u64 v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v));
}
__device__ __forceinline__ void st_word(unsigned *p, unsigned v) {
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v));
}

// ---- staging: bulk copies into shared memory, one mbarrier a buffer ------------
__device__ __forceinline__ void bar_init(unsigned bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_test(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bulk_load(unsigned dst, const void *src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void ld2(const double *p, double &x, double &y) {
    const double2 a = *reinterpret_cast<const double2 *>(p);
    x = a.x; y = a.y;
}
__device__ __forceinline__ void ld2(const float *p, float &x, float &y) {
    const float2 a = *reinterpret_cast<const float2 *>(p);
    x = a.x; y = a.y;
}
__device__ __forceinline__ void ld2(const int *p, int &x, int &y) {
    const int2 a = *reinterpret_cast<const int2 *>(p);
    x = a.x; y = a.y;
}
__device__ __forceinline__ void st2(double *p, double x, double y) {
    *reinterpret_cast<double2 *>(p) = make_double2(x, y);
}
__device__ __forceinline__ void st2(float *p, float x, float y) { *reinterpret_cast<float2 *>(p) = make_float2(x, y); }

template <int N> struct IntC { static constexpr int v = N; };

// one launch's tiles, components and hand-off words
template <class Real>
struct TileRun {
    SkewT<Real> g;
    unsigned mask;                  // the components of the launch
    Real *w;                        // the backward sweep's result (cell order), or null (g.w64)
    int N, ncc;                     // cells; components launched side by side (one bit of mask each)
    int *sync;
    typename Word<Real>::T *xfer;   // hand-off words: per component xstride of them
    long long xstride;
    long long maxSpin;
    int stall;                      // failure-detection test: the hand-off words never arrive
};

// staged arrays a chunk: MODE 2: D, Pz, Py, Px; MODE 0/1: the z, y, x
// coefficients and the right-hand side
constexpr int kStaged = 4;
constexpr int kWindow = 16;   // steps of hand-off words looked at together

// a CTA's shape and its ring: kRing steps of every tile's 32 results, then the
// ghosts: the last plane's results (TJ a tile) of the tiles before in k, and the
// last row's (TK a tile) of the tiles before in j.  A slot holds one step of
// the tile that formed the value.  A tile lags its producers by kSkewJ TJ or
// kSkewK TK steps, so the ring is deeper than that.
template <int TJ, int WJ, int WK>
struct Group {
    static constexpr int TK = 32 / TJ, W = WJ * WK;
    static constexpr int nK = TK > 1 ? WJ : 0, nJ = WK;   // streams of ghosts, and of results handed on
    static constexpr int ringSteps = TJ >= 32 ? 64 : 32;
    static constexpr int ghostK = 32 * W, ghostJ = ghostK + nK * TJ;
    static constexpr int pitch = (ghostJ + nJ * TK + 3) / 4 * 4;
    static constexpr int warps = 2 * W + 2 * (nK + nJ) + 1;
};

template <class Real, int P>
__host__ __device__ constexpr int stage_bytes() { return P * 32 * kStaged * (int)sizeof(Real); }
template <class Real, class G, int MODE, int P, int NB>
__host__ __device__ constexpr int group_smem() {   // (rD: a second ring, of the values' reciprocals)
    return G::W * NB * stage_bytes<Real, P>() + (MODE == 2 ? 2 : 1) * G::ringSteps * G::pitch * (int)sizeof(Real);
}

// counters shared by a CTA's warps (steps of a tile): computed and written out
// by each tile; ghosts that have arrived and results handed on by each stream;
// steps staged for each tile
enum { C_COMPUTED = 0, C_WRITTEN = 8, C_GHOST_K = 16, C_GHOST_J = 20, C_HANDED_K = 24, C_HANDED_J = 28, C_STAGED = 32, C_ABORT = 40,
       C_TICKET, C_COUNT };

// bounded wait until a counter reaches `need`, by all lanes; -1 when a wait ran out
template <int NS>
__device__ __forceinline__ int wait_steps(const volatile int *c, int need, volatile int *cnt, long long maxSpin) {
    long long spins = 0;
    int v;
    while ((v = __shfl_sync(0xffffffffu, *c, 0)) < need) {
        if ((++spins & 63) == 0 && (spins > maxSpin || cnt[C_ABORT])) {
            cnt[C_ABORT] = 1;
            return -1;
        }
        __nanosleep(NS);   // leaves the issue slots and the shared memory to the recurrence
    }
    return v;
}
// the lanes' counters until each has reached its need (the rare case, out of
// line: inlined it slows the recurrence's fast path down); the last values seen
__device__ __noinline__ int wait_watched(const volatile int *watch, int need, volatile int *cnt, long long maxSpin) {
    long long spins = 0;
    for (;;) {
        const int seen = *watch;
        if (__all_sync(0xffffffffu, seen >= need)) return seen;
        if ((++spins & 63) == 0 && (spins > maxSpin || cnt[C_ABORT])) {
            cnt[C_ABORT] = 1;
            return seen;
        }
    }
}
// lanes in step, without a barrier on the compiler's other memory accesses
__device__ __forceinline__ void warp_sync() { asm volatile("bar.warp.sync 0xffffffff;"); }

// MODE 0: forward application, 1: backward application, 2: rD recurrence
// (FP64 only).  The entry of (tile, step t, lane l) is tile * 32 T + (t / 2) *
// 64 + l * 2 + t % 2.  Entries outside the mesh have zero coefficients and
// right-hand sides, so every lane runs the same branch-free recurrence.
// The hand-off words of a tile: for each of its T steps the TJ results of its
// last plane, for the tile next in k, and the TK results of its last row, for
// the tile next in j.  Its step s is step s - offK (s - offJ) of that tile.
template <class Real, int MODE, int TJ, int WJ, int WK, int P, int NB>
__global__ void __launch_bounds__(32 * Group<TJ, WJ, WK>::warps, 1) k_tile_sweep(TileRun<Real> a) {
    typedef Group<TJ, WJ, WK> G;
    typedef Word<Real> Wd;
    typedef typename Wd::T W;
    constexpr int TK = 32 / TJ, PITCH = G::pitch, R = G::ringSteps;
    constexpr int offJ = kSkewJ * (TJ - 1), offK = kSkewK * (TK - 1);   // a producer's lead in steps
        constexpr int GS = sizeof(Real) == 8 ? 2 : 4;   // steps between two looks at the counters
    constexpr int B = 4;   // steps that share their slots' addresses
    static_assert(B % GS == 0 && P % B == 0 && P <= 16 && R % P == 0, "groups fill blocks, blocks chunks, chunks the ring");
    static_assert(kSkewJ * TJ % B == 0 && (TK == 1 || kSkewK * TK % B == 0), "a block of another tile's slots does not wrap");
    static_assert(kSkewJ == 1 && kSkewK == 1, "a step reads the values of the step before");
    constexpr W kNone = ~W(0);
    constexpr int RINV = R * PITCH;   // rD: a value's reciprocal in the second ring
    const Real zk = (MODE == 2) ? Real(1) : Real(0);
    SkewT<Real> &g = a.g;
    next_may_start();
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) u64 bars[G::W * NB];
    __shared__ int s_cnt[C_COUNT];
    volatile int *cnt = s_cnt;
    volatile Real *ring = reinterpret_cast<Real *>(smem + G::W * NB * stage_bytes<Real, P>());
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned bar0 = (unsigned)__cvta_generic_to_shared(bars);
    if (threadIdx.x == 0) {
        for (int i = 0; i < C_COUNT; ++i) s_cnt[i] = 0;
        for (int b = 0; b < G::W * NB; ++b) bar_init(bar0 + 8 * b);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    for (int i = threadIdx.x; i < (MODE == 2 ? 2 : 1) * R * PITCH; i += blockDim.x) ring[i] = zk;
    wait_for_previous();
    // every component of the launch has stopped iterating (the same word for
    // every CTA, written by an earlier kernel): nothing to do
    const unsigned live = g.dmask ? a.mask & *g.dmask : a.mask;
    if (!live) return;
    if (threadIdx.x == 0) s_cnt[C_TICKET] = atomicAdd(a.sync + SYNC_WORK, 1);
    __syncthreads();
    const int ticket = s_cnt[C_TICKET];
    // ticket t is group t / ncc of the (t % ncc)-th component, so every
    // component's groups are taken in dependency order
    unsigned m = a.mask;
    for (int q = ticket % a.ncc; q > 0; --q) m &= m - 1;
    const int comp = __ffs(m) - 1;
    if ((live >> comp) & 1u) {
        const int nTJ = g.nTJ, nTK = g.nTK, T = g.T;
        const int nGJ = (nTJ + WJ - 1) / WJ, grp = ticket / a.ncc;
        const int J0 = grp % nGJ * WJ, K0 = grp / nGJ * WK;   // the group's first tile, in the direction of the sweep
        // the role of this warp and its tile (or the tile at its stream's edge)
        int role, wj, wk;
        if (wid < 2 * G::W) {
            role = wid / G::W;   // 0 the recurrence, 1 results
            wj = wid % G::W % WJ;
            wk = wid % G::W / WJ;
        } else {
            const int q = wid - 2 * G::W;
            role = 2 + q / (G::nK + G::nJ);   // 2 ghosts, 3 results handed on, 4 staging
            const int st = q % (G::nK + G::nJ);
            const bool alongK = st < G::nK;
            if (role < 4) role += alongK ? 0 : 3;   // 5, 6: the same along j
            wj = alongK ? st : (role == 6 ? min(WJ, nTJ - J0) - 1 : 0);
            wk = alongK ? (role == 3 ? min(WK, nTK - K0) - 1 : 0) : st - G::nK;
            if (role == 4) {   // a lane a tile and array
                wj = lane / kStaged % WJ;
                wk = lane / kStaged / WJ % WK;
            }
        }
        const int w = wk * WJ + wj, J = J0 + wj, K = K0 + wk;
        const int here = K * nTJ + J;
        const int tile = (MODE == 1) ? (nTK - 1 - K) * nTJ + (nTJ - 1 - J) : here;
        const long long e0 = (long long)tile * T * 32;
        const int lf = (MODE == 1) ? 31 - lane : lane;   // the lane's column in the forward layout
        const bool there = J < nTJ && K < nTK && !(role == 4 && lane >= kStaged * G::W), exists = there || role == 4;
        // hand-off words: [tile][T][TJ] along k, then [tile][T][TK] along j
        W *xk = a.xfer + (long long)comp * a.xstride, *xj = xk + (long long)nTJ * nTK * T * TJ;
        const long long maxLocal = a.maxSpin << 7;   // spins on shared memory: shorter, and never the first to run out
        const unsigned myBars = bar0 + 8 * w * NB;
        unsigned char *myStage = smem + (size_t)w * NB * stage_bytes<Real, P>();
        if (!exists) {
        } else if (role == 0) {
            // ---- the recurrence -------------------------------------------------
            const int lj = lane % TJ, lk = lane / TJ;
            // where this lane's neighbours' values are in a slot, and whether they
            // are another tile's (a slot kSkew? * T? steps on)
            // (in one plane the k coefficients are zero: any value serves)
            const bool farK = TK > 1 && lk == 0, farJ = lj == 0;
            const int iK = TK == 1 ? w * 32 + lane
                           : !farK ? w * 32 + lane - TJ
                           : wk > 0 ? (w - WJ) * 32 + (TK - 1) * TJ + lj
                                    : G::ghostK + wj * TJ + lj;
            const int iJ = !farJ ? w * 32 + lane - 1
                           : wj > 0 ? (w - 1) * 32 + lk * TJ + TJ - 1
                                    : G::ghostJ + wk * TK + lk;
            const int leadK = farK ? kSkewK * TK : 0, leadJ = farJ ? kSkewJ * TJ : 0;
            // what must have happened before a group of steps t .. t + GS - 1:
            // lanes 0 .. 4 each watch a counter that must reach min(t + off, T)
            const volatile int *watch = cnt + C_COMPUTED + w;
            int off = -(1 << 29);
            if (lane == 0 && (wj > 0 || J > 0)) {   // the j producer's steps
                watch = wj > 0 ? cnt + C_COMPUTED + w - 1 : cnt + C_GHOST_J + wk;
                off = GS + offJ;
            } else if (lane == 1 && (wk > 0 || (TK > 1 && K > 0))) {   // the k producer's
                watch = wk > 0 ? cnt + C_COMPUTED + w - WJ : cnt + C_GHOST_K + wj;
                off = GS + offK;
            } else if (lane == 2 && J + 1 < nTJ) {   // the j consumer has read what these steps overwrite
                watch = wj + 1 < WJ ? cnt + C_COMPUTED + w + 1 : cnt + C_HANDED_J + wk;
                off = GS - R;
            } else if (lane == 3 && TK > 1 && K + 1 < nTK) {
                watch = wk + 1 < WK ? cnt + C_COMPUTED + w + WJ : cnt + C_HANDED_K + wj;
                off = GS - R;
            } else if (lane == 4) {
                watch = cnt + C_WRITTEN + w;
                off = GS - R;
            } else if (lane == 5) {   // the coefficients (a chunk arrives whole)
                watch = cnt + C_STAGED + w;
                off = GS;
            }
            int seen = 0;
            Real y1 = zk, inv1 = zk;
            // looks at the counters until the steps from t on may be taken
            auto until_ready = [&](int t) {
                const int need = min(t + off, T);
                if (!__all_sync(0xffffffffu, seen >= need)) seen = wait_watched(watch, need, cnt, maxLocal);
            };
            int buf = 0;
            for (int t0 = 0; t0 < T; t0 += P) {
                until_ready(t0);
                const Real *db = reinterpret_cast<const Real *>(myStage + (size_t)buf * stage_bytes<Real, P>());
                Real va[kStaged][P];
#pragma unroll
                for (int i = 0; i < kStaged; ++i)
#pragma unroll
                    for (int s = 0; s < P; s += 2) ld2(db + i * P * 32 + s * 32 + lf * 2, va[i][s], va[i][s + 1]);
#pragma unroll
                for (int b0 = 0; b0 < P; b0 += B) {
                    const int tb = t0 + b0;
                    volatile Real *cur = ring + (tb & (R - 1)) * PITCH + w * 32 + lane;
                    // the neighbours' slots of step tb - 1 and from tb on
                    const volatile Real *kPast = ring + ((tb - 1 + leadK) & (R - 1)) * PITCH + iK;
                    const volatile Real *kNow = ring + ((tb + leadK) & (R - 1)) * PITCH + iK;
                    const volatile Real *jPast = ring + ((tb - 1 + leadJ) & (R - 1)) * PITCH + iJ;
                    const volatile Real *jNow = ring + ((tb + leadJ) & (R - 1)) * PITCH + iJ;
#pragma unroll
                    for (int s = 0; s < B; ++s) {
                        if (s % GS == 0) {
                            if (b0 + s > 0) until_ready(tb + s);
                            seen = *watch;   // for the next group
                        }
                        const int sf = (MODE == 1) ? P - 1 - b0 - s : b0 + s;
                        const Real xz = s >= 1 ? kNow[(s - 1) * PITCH] : kPast[0];
                        const Real xy = s >= 1 ? jNow[(s - 1) * PITCH] : jPast[0];
                        Real v;
                        if constexpr (MODE == 2) {   // D - Pz / rD(k-1) - Py / rD(j-1) - Px / rD(i-1)
                            const Real iz = s >= 1 ? kNow[RINV + (s - 1) * PITCH] : kPast[RINV];
                            const Real iy = s >= 1 ? jNow[RINV + (s - 1) * PITCH] : jPast[RINV];
                            v = r_sub(va[0][sf], quotient(va[1][sf], divisor(xz, iz)));
                            v = r_sub(v, quotient(va[2][sf], divisor(xy, iy)));
                            v = r_sub(v, quotient(va[3][sf], divisor(y1, inv1)));
                            inv1 = __drcp_rn(v);
                            cur[RINV + s * PITCH] = inv1;
                        } else {
                            v = r_fma(-va[0][sf], xz, va[3][sf]);
                            if (sizeof(Real) == 4) {
                                // FP32: the i term before the j term
                                v = r_fma(-va[2][sf], y1, v);
                                v = r_fma(-va[1][sf], xy, v);
                            } else {
                                v = r_fma(-va[1][sf], xy, v);
                                v = r_fma(-va[2][sf], y1, v);
                            }
                        }
                        cur[s * PITCH] = v;
                        y1 = v;
                        warp_sync();
                        if (s % 2 == 1) cnt[C_COMPUTED + w] = tb + s + 1;   // (every lane the same word)
                    }
                }
                if (cnt[C_ABORT]) break;
                if (++buf == NB) buf = 0;
            }
        } else if (role == 1) {
            // ---- results out -----------------------------------------------------
            auto first = [&](int tc) { return e0 + (long long)((MODE == 1) ? T - tc - P : tc) * 32; };
            int cell[MODE == 1 ? P : 2], next[MODE == 1 ? P : 2];
            auto cells = [&](int at) {   // of the chunk from step at on
                if (MODE == 1 && at < T) {
#pragma unroll
                    for (int s = 0; s < P; s += 2) ld2(g.cellOf + first(at) + s * 32 + lf * 2, next[s], next[s + 1]);
                }
            };
            cells(0);
            for (int at = 0; at < T; at += P) {
                if (MODE == 1) {
#pragma unroll
                    for (int s = 0; s < P; ++s) cell[s] = next[s];
                    cells(at + P);   // before the wait
                }
                if (wait_steps<100>(cnt + C_COMPUTED + w, at + P, cnt, maxLocal) < 0) break;
                const volatile Real *res = ring + (at & (R - 1)) * PITCH + w * 32 + lane;
                Real out[P];
#pragma unroll
                for (int s = 0; s < P; ++s) out[s] = res[s * PITCH];
                __syncwarp();
                cnt[C_WRITTEN + w] = at + P;   // (read: the ring may take the next steps)
                if (MODE == 1) {
                    if (g.w64) {
#pragma unroll
                        for (int s = 0; s < P; ++s)
                            if (cell[P - 1 - s] >= 0) g.w64[(long long)comp * a.N + cell[P - 1 - s]] = (double)out[s];
                    } else {
#pragma unroll
                        for (int s = 0; s < P; ++s)
                            if (cell[P - 1 - s] >= 0) a.w[(long long)comp * a.N + cell[P - 1 - s]] = out[s];
                    }
                } else {
                    Real *dst = ((MODE == 2) ? g.rDraw : g.wS + (long long)comp * g.nSkew) + first(at) + lane * 2;
#pragma unroll
                    for (int s = 0; s < P; s += 2) st2(dst + s * 32, out[s], out[s + 1]);
                }
            }
        } else if (role == 4) {
            // ---- coefficients in: a lane a tile and array ---------------------------
            const int array = lane % kStaged;
            const Real *src;
            if (MODE == 2) {
                src = array == 0 ? g.D : array == 1 ? g.Pz : array == 2 ? g.Py : g.Px;
            } else {
                src = array == 0   ? (MODE == 0 ? g.Az : g.Bz)
                      : array == 1 ? (MODE == 0 ? g.Ay : g.By)
                      : array == 2 ? (MODE == 0 ? g.Ax : g.Bx)
                                   : (MODE == 0 ? g.rS : g.wS) + (long long)comp * g.nSkew;
            }
            const unsigned dst = (unsigned)__cvta_generic_to_shared(myStage) + array * P * 32 * (int)sizeof(Real);
            const bool leads = array == 0;
            // steps in flight, in order, and told to the recurrence as they arrive
            int staged = there ? 0 : T, told = staged;
            long long spins = 0;
            while (__any_sync(0xffffffffu, told < T)) {
                // (a buffer is free once its last chunk has been computed)
                bool go = staged < T && !cnt[C_ABORT] && cnt[C_COMPUTED + w] >= staged - (NB - 1) * P;
                go = __shfl_sync(0xffffffffu, go, lane & ~(kStaged - 1));
                const int b = staged / P % NB;
                if (go && leads) bar_expect(myBars + 8 * b, stage_bytes<Real, P>());
                __syncwarp();
                if (go) {
                    const long long lo = e0 + (long long)((MODE == 1) ? T - staged - P : staged) * 32;
                    bulk_load(dst + b * stage_bytes<Real, P>(), src + lo, P * 32 * sizeof(Real), myBars + 8 * b);
                    staged += P;
                }
                if (told < staged && bar_test(myBars + 8 * (told / P % NB), (told / P / NB) & 1)) {
                    told += P;
                    if (leads) cnt[C_STAGED + w] = told;
                    spins = 0;
                }
                if ((++spins & 63) == 0 && (spins > maxLocal || cnt[C_ABORT])) {
                    cnt[C_ABORT] = 1;
                    if (told == staged) told = staged = T;   // given up, with no copy in flight
                }
            }
        } else if (role == 2 || role == 5) {
            // ---- ghosts: one stream, from the tile before in k (j) to tile w -------
            auto ghosts = [&](auto nConst, int off, W *src, int ringAt, volatile int *arrived, bool any) {
                constexpr int n = decltype(nConst)::v;            // words a step
                constexpr int L = (kWindow * n + 31) / 32;        // and words a lane
                int pos = any ? off : T;                          // the producer's step
                if (!any) return;
                long long spins = 0;
                while (pos < T) {
                    // the ring holds the producer's steps before `room`
                    const int room = min(T, __shfl_sync(0xffffffffu, cnt[C_COMPUTED + w], 0) + R);
                    W v[L];
#pragma unroll
                    for (int i = 0; i < L; ++i) {
                        const int q = i * 32 + lane, st = pos + q / n;
                        v[i] = q < kWindow * n && st < room ? ld_word(src + (long long)st * n + q % n) : kNone;
                    }
                    // whole steps that have arrived
                    int k = kWindow * n;
#pragma unroll
                    for (int i = L - 1; i >= 0; --i) {
                        const unsigned no = __ballot_sync(0xffffffffu, v[i] == kNone);
                        if (no) k = i * 32 + __ffs(no) - 1;
                    }
                    k = a.stall ? 0 : min(k, kWindow * n) / n;
                    if (k == 0) {
                        if ((++spins & 63) == 0 &&
                            (spins > a.maxSpin || cnt[C_ABORT] || *(volatile int *)(a.sync + SYNC_ERROR))) {
                            cnt[C_ABORT] = 1;
                            break;
                        }
                        continue;
                    }
                    spins = 0;
#pragma unroll
                    for (int i = 0; i < L; ++i) {
                        const int q = i * 32 + lane, st = pos + q / n;
                        if (st < pos + k) {
                            volatile Real *to = ring + (st & (R - 1)) * PITCH + ringAt + q % n;
                            to[0] = Wd::value(v[i]);
                            if constexpr (MODE == 2) to[RINV] = __drcp_rn(Wd::value(v[i]));
                        }
                    }
                    __syncwarp();
                    *arrived = pos + k;
#pragma unroll
                    for (int i = 0; i < L; ++i) {
                        const int q = i * 32 + lane, st = pos + q / n;
                        if (st < pos + k) st_word(src + (long long)st * n + q % n, kNone);
                    }
                    pos += k;
                }
            };
            if (role == 2)
                ghosts(IntC<TJ>{}, offK, xk + (long long)(here - nTJ) * T * TJ, G::ghostK + wj * TJ, cnt + C_GHOST_K + wj,
                       K > 0);
            else
                ghosts(IntC<TK>{}, offJ, xj + (long long)(here - 1) * T * TK, G::ghostJ + wk * TK, cnt + C_GHOST_J + wk,
                       J > 0);
        } else {
            // ---- one stream of results handed on, from tile w ----------------------
            auto hand_on = [&](auto nConst, W *dst, int ringAt, int stride, volatile int *handed, bool any) {
                constexpr int n = decltype(nConst)::v;
                constexpr int L = (kWindow * n + 31) / 32;
                if (!any) return;
                int pos = 0;
                while (pos < T) {
                    const int c = wait_steps<20>(cnt + C_COMPUTED + w, pos + 1, cnt, maxLocal);
                    if (c < 0) break;
                    const int k = min(c - pos, kWindow);
#pragma unroll
                    for (int i = 0; i < L; ++i) {
                        const int q = i * 32 + lane, st = pos + q / n;
                        if (st < pos + k) {
                            const W v = Wd::of(ring[(st & (R - 1)) * PITCH + ringAt + q % n * stride]);
                            st_word(dst + (long long)st * n + q % n, v == kNone ? Wd::kOtherNaN : v);
                        }
                    }
                    pos += k;
                    __syncwarp();
                    *handed = pos;
                }
            };
            if (role == 3)
                hand_on(IntC<TJ>{}, xk + (long long)here * T * TJ, w * 32 + 32 - TJ, 1, cnt + C_HANDED_K + wj, K + 1 < nTK);
            else
                hand_on(IntC<TK>{}, xj + (long long)here * T * TK, w * 32 + TJ - 1, TJ, cnt + C_HANDED_J + wk, J + 1 < nTJ);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (cnt[C_ABORT]) atomicExch(a.sync + SYNC_ERROR, 1);
        // the last CTA to finish re-arms the counters for the next launch
        const int n = atomicAdd(a.sync + SYNC_DONE, 1);
        if (n == (int)gridDim.x - 1) {
            a.sync[SYNC_WORK] = 0;
            a.sync[SYNC_DONE] = 0;
        }
    }
}

// rS = rD r gathered into the skewed layout (0 outside the mesh): the first
// product of the forward recurrence, rounded as the sequential sweep rounds it
// (an FP64 right-hand side of the FP32 sweeps is rounded first)
template <class Real, class In>
__device__ __forceinline__ void k_skew_gather_body(SkewT<Real> g, unsigned mask, int nc, const In *__restrict__ r, int
                                                  N) {
    long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= g.nSkew) return;
    if (g.dmask) mask &= *g.dmask;
    int c = g.cellOf[e];
    const Real rd = g.rDinv[e];
    for (int q = 0; q < nc; ++q)
        if ((mask >> q) & 1u)
            g.rS[(long long)q * g.nSkew + e] = c >= 0 ? r_mul(rd, (Real)r[(long long)q * N + c]) : Real(0);
}
template <class Real, class In>
__global__ void k_skew_gather(SkewT<Real> g, unsigned mask, int nc, const In *r, int N) {
    after_previous();
    k_skew_gather_body<Real, In>(g, mask, nc, r, N);
}

// gather the skewed per-entry coefficients of one matrix
__global__ void k_skew_setup(SkewView g, const int *__restrict__ faceLo, int N, const double *__restrict__ diag,
                             const double *__restrict__ upper, const double *__restrict__ lower) {
    long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= g.nSkew) return;
    int c = g.cellOf[e];
    double d = 1.0, pz = 0.0, py = 0.0, px = 0.0;
    if (c >= 0) {
        d = diag[c];
        int fz = faceLo[c], fy = faceLo[N + c], fx = faceLo[2 * N + c];
        if (fz >= 0) pz = __dmul_rn(upper[fz], lower[fz]);
        if (fy >= 0) py = __dmul_rn(upper[fy], lower[fy]);
        if (fx >= 0) px = __dmul_rn(upper[fx], lower[fx]);
    }
    g.D[e] = d;
    g.Pz[e] = pz;
    g.Py[e] = py;
    g.Px[e] = px;
}

// rD -> 1/rD and the premultiplied sweep coefficients rD_c a_cf
__global__ void k_skew_premul(SkewView g, const int *__restrict__ faceLo, const int *__restrict__ faceHi, int N,
                              const double *__restrict__ upper, const double *__restrict__ lower) {
    long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= g.nSkew) return;
    int c = g.cellOf[e];
    double rd = 0.0, az = 0.0, ay = 0.0, ax = 0.0, bz = 0.0, by = 0.0, bx = 0.0;
    if (c >= 0) {
        rd = 1.0 / g.rDraw[e];
        int fz = faceLo[c], fy = faceLo[N + c], fx = faceLo[2 * N + c];
        int gz = faceHi[c], gy = faceHi[N + c], gx = faceHi[2 * N + c];
        if (fz >= 0) az = rd * lower[fz];
        if (fy >= 0) ay = rd * lower[fy];
        if (fx >= 0) ax = rd * lower[fx];
        if (gz >= 0) bz = rd * upper[gz];
        if (gy >= 0) by = rd * upper[gy];
        if (gx >= 0) bx = rd * upper[gx];
    }
    g.rDinv[e] = rd;
    g.Az[e] = az; g.Ay[e] = ay; g.Ax[e] = ax;
    g.Bz[e] = bz; g.By[e] = by; g.Bx[e] = bx;
}

// FP32 copies of the FP64 sweep coefficients
__global__ void k_skew_to32(SkewView g, SkewView32 h) {
    long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= g.nSkew) return;
    h.rDinv[e] = (float)g.rDinv[e];
    h.Az[e] = (float)g.Az[e]; h.Ay[e] = (float)g.Ay[e]; h.Ax[e] = (float)g.Ax[e];
    h.Bz[e] = (float)g.Bz[e]; h.By[e] = (float)g.By[e]; h.Bx[e] = (float)g.Bx[e];
}

namespace {

// the hand-off words of ncomp components, all ones, kept per precision (the
// words that no consumer reads keep old values, at the same places in every
// launch of that precision)
template <class Real>
typename Word<Real>::T *hand_off_words(rt_ctx *ctx, long long perComp, int ncomp) {
    StructMesh &s = ctx->mesh.sm;
    DBuf<u64> &buf = s.xfer[sizeof(Real) == 4 ? 1 : 0];
    const size_t need = ((size_t)perComp * ncomp * sizeof(Real) + 7) / 8;
    if (buf.n < need) {
        buf.alloc(need);
        RT_CUDA(cudaMemsetAsync(buf.p, 0xff, buf.n * 8, ctx->stream));
    }
    return reinterpret_cast<typename Word<Real>::T *>(buf.p);
}

template <class Real, int MODE, int TJ, int WJ, int WK, int P, int NB>
void launch_one(rt_ctx *ctx, const TileRun<Real> &run) {
    typedef Group<TJ, WJ, WK> G;
    constexpr int shm = group_smem<Real, G, MODE, P, NB>();
    static_assert(shm <= 226 * 1024, "one CTA's shared memory");
    // (the current device's attribute: set at each launch, for contexts on any device)
    RT_CUDA(cudaFuncSetAttribute(k_tile_sweep<Real, MODE, TJ, WJ, WK, P, NB>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
    const int groups = (run.g.nTJ + WJ - 1) / WJ * ((run.g.nTK + WK - 1) / WK);
    launch_next(k_tile_sweep<Real, MODE, TJ, WJ, WK, P, NB>, groups * run.ncc, 32 * G::warps, shm, ctx->stream, run);
}

// Schedules of the sweeps (sweep.h): chunk size P (steps per staged block), staging
// depth NB (blocks in flight) and with them the CTA's tiles: chunks of 16 steps leave
// an FP64 CTA room for two.  RT_OPT_SWEEP_TUNE takes one of them; the default is
// two tiles and (16, 3), as fewer warps share the SM's issue slots (1M cells,
// one component: FP64 235 us an application against 248 with four tiles and
// (8, 5), FP32 132 against 154), but four when the groups of two would not all
// run at once, one an SM (three components: FP64 258 us against 330, FP32 162
// against 169).
constexpr int kNarrow = 2, kWide = 1;

template <class Real, int MODE, int TJ>
void launch_tuned(rt_ctx *ctx, const TileRun<Real> &run, bool all, int k) {
    if constexpr (MODE == 2) {   // its two rings leave room for these
        if constexpr (TJ == 8) {
            if (!all) return launch_one<Real, MODE, TJ, 2, 2, 8, 3>(ctx, run);
        }
        launch_one<Real, MODE, TJ, 2, 1, 16, 3>(ctx, run);
    } else {
        constexpr int WJ = TJ == 32 ? 4 : 2, WK = TJ == 32 ? 1 : 2;
        switch (k) {
        case 0: launch_one<Real, MODE, TJ, WJ, WK, kTuneP[0], kTuneNB[0]>(ctx, run); break;
        case 1: launch_one<Real, MODE, TJ, WJ, WK, kTuneP[1], kTuneNB[1]>(ctx, run); break;
        case 2: launch_one<Real, MODE, TJ, 2, 1, kTuneP[2], kTuneNB[2]>(ctx, run); break;
        case 3: launch_one<Real, MODE, TJ, 2, 1, kTuneP[3], kTuneNB[3]>(ctx, run); break;
        default: launch_one<Real, MODE, TJ, WJ, WK, kTuneP[4], kTuneNB[4]>(ctx, run); break;
        }
    }
}

// one sweep of the masked components, side by side in one launch
template <class Real, int MODE>
void launch_mode(rt_ctx *ctx, const SkewT<Real> &g, unsigned mask, Real *w) {
    StructMesh &s = ctx->mesh.sm;
    if (!mask) return;
    TileRun<Real> run;
    run.g = g;
    run.mask = mask;
    run.w = w;
    run.N = ctx->mesh.N;
    run.ncc = __builtin_popcount(mask);
    run.sync = s.sync.p;
    run.xstride = (long long)s.nTJ * s.nTK * (s.TJ + 32 / s.TJ) * s.T;
    run.xfer = hand_off_words<Real>(ctx, run.xstride, 32 - __builtin_clz(mask));
    // a spin is an L2 round trip: 2^24 / 8 of them are about a second
    run.maxSpin = std::max(64ll, ctx->waitLimit >> 3);
    run.stall = ctx->stallTest > 0 ? 1 : 0;
    if (run.stall) --ctx->stallTest;
    const bool all = (s.nTJ + 1) / 2 * s.nTK * run.ncc <= ctx->numSMs;   // groups of two tiles, one an SM
    const int k = ctx->sweepTune > 0 ? ctx->sweepTune - 1 : all ? kNarrow : kWide;
    if (MODE != 2) s.tune[sizeof(Real) == 4 ? 1 : 0] = k;
    if (s.TJ == 32) launch_tuned<Real, MODE, 32>(ctx, run, all, k);
    else launch_tuned<Real, MODE, 8>(ctx, run, all, k);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
    s.pendingCheck = true;
}

}  // namespace

void skew_prepare(rt_ctx *ctx, const double *diag, const double *upper, const double *lower) {
    StructMesh &s = ctx->mesh.sm;
    SkewView g = s.view();
    int nb = nblocks(g.nSkew);
    k_skew_setup<<<nb, RT_BLOCK, 0, ctx->stream>>>(g, s.faceLo.p, ctx->mesh.N, diag, upper, lower);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
    launch_mode<double, 2>(ctx, g, 1u, (double *)nullptr);
    k_skew_premul<<<nb, RT_BLOCK, 0, ctx->stream>>>(g, s.faceLo.p, s.faceHi.p, ctx->mesh.N, upper, lower);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
}

void skew_precondition(rt_ctx *ctx, int nc, unsigned mask, const double *r, double *w, const unsigned *dmask) {
    SkewView g = ctx->mesh.sm.view();
    g.dmask = dmask;
    launch_next(k_skew_gather<double, double>, nblocks(g.nSkew), RT_BLOCK, 0, ctx->stream, g, mask, nc, r, ctx->mesh.N);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
    launch_mode<double, 0>(ctx, g, mask, w);
    launch_mode<double, 1>(ctx, g, mask, w);
}

// 1/rD of the last skew_prepare, in cell order
__global__ void k_skew_rdinv_cells(SkewView g, double *__restrict__ rDc) {
    long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= g.nSkew) return;
    const int c = g.cellOf[e];
    if (c >= 0) rDc[c] = g.rDinv[e];
}

void skew_rdinv_cells(rt_ctx *ctx, double *rDc) {
    SkewView g = ctx->mesh.sm.view();
    k_skew_rdinv_cells<<<nblocks(g.nSkew), RT_BLOCK, 0, ctx->stream>>>(g, rDc);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
}

void skew_prepare_T(rt_ctx *ctx, const double *upper, const double *lower) {
    StructMesh &s = ctx->mesh.sm;
    SkewView g = s.viewT();
    // the lower and upper coefficients exchanged: forward sweep rD_c a_fc,
    // backward rD_c a_cf (rDinv is rewritten with the same values)
    k_skew_premul<<<nblocks(g.nSkew), RT_BLOCK, 0, ctx->stream>>>(g, s.faceLo.p, s.faceHi.p, ctx->mesh.N, lower,
                                                                  upper);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
}

void skew_precondition_T(rt_ctx *ctx, int nc, unsigned mask, const double *r, double *w) {
    SkewView g = ctx->mesh.sm.viewT();
    launch_next(k_skew_gather<double, double>, nblocks(g.nSkew), RT_BLOCK, 0, ctx->stream, g, mask, nc, r, ctx->mesh.N);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
    launch_mode<double, 0>(ctx, g, mask, w);
    launch_mode<double, 1>(ctx, g, mask, w);
}

void skew_prepare32(rt_ctx *ctx, const double *diag, const double *upper, const double *lower) {
    skew_prepare(ctx, diag, upper, lower);
    StructMesh &s = ctx->mesh.sm;
    SkewView g = s.view();
    SkewView32 h = s.view32();
    k_skew_to32<<<nblocks(g.nSkew), RT_BLOCK, 0, ctx->stream>>>(g, h);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
}

void skew_precondition32(rt_ctx *ctx, int nc, unsigned mask, const float *r, float *w, const unsigned *dmask) {
    SkewView32 g = ctx->mesh.sm.view32();
    g.dmask = dmask;
    launch_next(k_skew_gather<float, float>, nblocks(g.nSkew), RT_BLOCK, 0, ctx->stream, g, mask, nc, r, ctx->mesh.N);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
    launch_mode<float, 0>(ctx, g, mask, w);
    launch_mode<float, 1>(ctx, g, mask, w);
}

void skew_precondition32d(rt_ctx *ctx, int nc, unsigned mask, const double *r, double *w, const unsigned *dmask) {
    SkewView32 g = ctx->mesh.sm.view32();
    g.w64 = w;
    g.dmask = dmask;
    launch_next(k_skew_gather<float, double>, nblocks(g.nSkew), RT_BLOCK, 0, ctx->stream, g, mask, nc, r, ctx->mesh.N);
    RT_CHECK_LAUNCH();
    launch_count(ctx);
    launch_mode<float, 0>(ctx, g, mask, (float *)nullptr);
    launch_mode<float, 1>(ctx, g, mask, (float *)nullptr);
}

rt_status skew_check(rt_ctx *ctx) {
    StructMesh &s = ctx->mesh.sm;
    if (!s.pendingCheck) return RT_OK;
    int err = 0;
    RT_CUDA(cudaMemcpyAsync(&err, s.sync.p + SYNC_ERROR, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    RT_CUDA(cudaStreamSynchronize(ctx->stream));
    s.pendingCheck = false;
    if (err) {   // words were left behind and unread: clear them all
        RT_CUDA(cudaMemsetAsync(s.sync.p, 0, sizeof(int) * SYNC_WORDS, ctx->stream));
        for (DBuf<u64> &x : s.xfer)
            if (x.p) RT_CUDA(cudaMemsetAsync(x.p, 0xff, x.n * 8, ctx->stream));
    }
    return err ? RT_ETIMEOUT : RT_OK;
}

}  // namespace rt
