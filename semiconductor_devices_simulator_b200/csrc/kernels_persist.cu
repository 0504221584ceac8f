// Persistent linear solves: one cooperative launch runs a whole multigrid-preconditioned
// Krylov solve of an instance - the hierarchy set-up, every iteration, both V-cycles of a
// BiCGSTAB iteration, and for the refined path every FP64 refinement step around its FP32
// inner solves - with grid-wide barriers between the dependent passes instead of kernel
// boundaries.
//
// What bounds it: a V-cycle is a chain of dependent half sweeps, each a pass over a part of
// one level that is resident in the L2 (below ~1M nodes), so a solve costs (passes) x
// (barrier + one pass's latency and L2 traffic).  The layout and the passes are built for that:
//   * the solve keeps its own copy of every level, colour by colour (SLev, semisim.h): a half
//     sweep reads its couplings, pivots and right-hand side as contiguous pairs and the other
//     colour's values as contiguous pairs too.  In the natural order every sector of a half
//     sweep is half unused (576,000 nodes, FP32: a finest-level pass takes 2.3 us, 4.2 us in the
//     natural order with 1024 threads);
//   * the red-black D-ILU application is written as red solve / black update with the D-ILU
//     pivot / red solve.  Red rows are then exact after every application, so no residual array
//     is kept: the restriction sums black residuals only, the way up needs no residual pass
//     (its first red solve reads the prolonged black values), and A M^-1 b on red rows is b itself;
//   * whoever writes a right-hand side also writes the first red values D b, so the first black
//     half sweep reads them directly;
//   * the BiCGSTAB iteration's rho comes from the two dot products rh.s and rh.t taken with the
//     passes before, so x, r and the next p are updated in one pass; PCG takes its step length
//     from z.A z and the recurrence q = A z + beta q, with one reduction per iteration.
//
// Layout of the work:
//   * every block runs the passes of the large levels (0 .. Ls-1) as grid-stride loops
//     over the pass's index space, one barrier after each pass;
//   * block 0 keeps the small levels (Ls .. coarsest) in its shared memory for the whole
//     solve and runs their part of every V-cycle with barriers of as many warps as the level
//     has work for, while the other blocks wait at the next grid barrier;
//   * reductions: each block writes its partial record, and after the barrier every block
//     sums all records in block order, so every block holds bit-identical totals and takes
//     the same stop decisions with no extra barrier.
//
// The stop rules are the reference's (pcg semiconductor_3d.c:2182-2210, bicgstab_core
// :2234-2320) as the per-pass path applies them, and the refinement the same FP64 rule.
//
// Safety: the launch is cooperative (all blocks co-resident).  Every wait at a grid barrier is
// bounded: after 2 s a block sets the error word and leaves, every other block
// leaves at its next wait, and the host restores the solve's start and repeats it on the
// per-pass path.  The cluster barriers (one-cluster grids, and the coarse levels in the first
// cluster) are the hardware's and have no limit: a cluster is scheduled as a whole, its blocks
// pass the same barriers between two grid barriers, and blocks that have left are not waited for.
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <mutex>
#include <vector>

#include "la_common.cuh"
#include "persist_common.cuh"
#include "prof.h"

// the pass functions inline into the kernel (compiled apart, __noinline__, they measured
// 30 % slower: every view field was reloaded after each store)
#ifndef PG_PASS
#define PG_PASS __forceinline__
#endif

// the set-up functions are shared by the large levels and block 0's small ones: code met for
// the first time in a launch is fetched from L2 line by line (the small levels' own inlined
// copies took 5 us each there, 0.7 us warm)
#define PG_SETUP __noinline__

namespace ss {

// 512 threads of 128 registers: with 1024 of 64 the half sweeps' operands spilled to local
// memory, which every barrier's acquire throws out of the L1 (a BiCGSTAB solve of the
// 576,000-node MOSFET: 1278 us with 1024 threads, 1035 us with 512, FP64 1586 and 1095 us)
constexpr int PT_TPB = 512;

enum PKind { PK_PCG = 0, PK_BICG = 1, PK_REFINED = 2 };

struct PArgs {
    int Ls;          // first level of the shared-memory part (>= 1)
    int deep;        // levels (from the finest) with two smoother applications
    int sweeps2;     // 1: the second application is on
    int maxsteps;    // refinement steps at most (PK_REFINED)
    int qsign;       // Slotboom weights of the hierarchy: 0 none (Poisson), +1 electrons, -1 holes
    unsigned long long *trace;   // barrier timeline of this launch (null: off)
    int ntrace;
    int barmode;                 // grid-barrier form (persist_common.cuh)
    int csz;                     // CTAs of a thread-block cluster (0: launched without clusters)
    int Lc;                      // first level the first cluster runs alone (cluster barriers)
    int onecl;                   // the whole grid is one cluster
    double alpha;    // prolongation factor
    double rtol, atol;   // stop rule of the FP64 BiCGSTAB start (PK_BICG)
    KrylovS rec[2];      // starting records: the loop's, and the refinement's (PK_REFINED)
};

// ---------------------------------------------------------------- layout on the host
// 256-byte aligned arrays of every level and the level-0 vectors, from `base`
template <class T>
size_t persist_work_layout(char *base, const int dims[][6], int nlev, SWork<T> *w) {
    size_t off = 0;
    auto take = [&](size_t n) {
        T *p = base ? reinterpret_cast<T *>(base + off) : nullptr;
        off += (n * sizeof(T) + 255) & ~size_t(255);
        return p;
    };
    for (int L = 0; L < nlev; L++) {
        SLev<T> v{};
        v.Nx = dims[L][0]; v.Ny = dims[L][1]; v.Nz = dims[L][2];
        v.N = v.Nx * v.Ny * v.Nz;
        v.cx = dims[L][3]; v.cy = dims[L][4]; v.cz = dims[L][5];
        v.last = L == nlev - 1;
        v.hx = (((v.Nx + 1) / 2) + 1) & ~1;
        v.sz = v.hx * v.Ny;
        v.H = v.sz * v.Nz;
        v.ap = (2 * v.H + 31) & ~31;
        v.n8 = (v.Nx + 7) / 8;
        v.fr = fast_div(v.hx / 2);
        v.fy = fast_div(v.Ny);
        v.f8 = fast_div(v.n8);
        v.A = take((size_t)6 * v.ap);
        v.G = take((size_t)2 * v.H);
        v.D = take(v.last ? std::max((size_t)2 * v.H, (size_t)COARSE_MAX * COARSE_MAX) : (size_t)2 * v.H);
        v.pw = take((size_t)2 * v.H);
        if (L) { v.x = take((size_t)2 * v.H); v.b = take((size_t)2 * v.H); }
        if (w) w->lev[L] = v;
    }
    const size_t n0 = 2 * (size_t)(((((dims[0][0] + 1) / 2) + 1) & ~1)) * dims[0][1] * dims[0][2];
    for (int q = 0; q < PW_VEC; q++) { T *p = take(n0); if (w) w->vec[q] = p; }
    T *p = take(n0);
    if (w) w->w0 = p;
    return off;
}
template size_t persist_work_layout<double>(char *, const int[][6], int, SWork<double> *);
template size_t persist_work_layout<float>(char *, const int[][6], int, SWork<float> *);

// ---------------------------------------------------------------- on-chip tables
template <class T> __device__ __forceinline__ const SWork<T> *swork(const DevP &P);
template <> __device__ __forceinline__ const SWork<double> *swork<double>(const DevP &P) { return P.pwd; }
template <> __device__ __forceinline__ const SWork<float> *swork<float>(const DevP &P) { return P.pwf; }

// Every descriptor a pass needs is copied into shared memory once per launch: after each
// grid barrier the acquire invalidates L1, so a descriptor read from global memory would
// cost a chain of dependent L2 round trips per pass.
template <class T>
struct PTab {
    SWork<T> w;
    SLev<T> sv[MAXLEV];          // block 0: the levels it keeps in shared memory (index L - Ls)
    int slot[COARSE_MAX];        // block 0: the coarsest level's slots in the order of its dense inverse's rows
    int cslot[COARSE_MAX];       // and in the order of its columns
    SLev<T> cur0;                // level 0 with the running V-cycle's b and x
    const double *A64;           // the FP64 level-0 operator in natural order (coupling q at A64 + q * ap64 + k)
    int ap64;
};
// level 0 with the V-cycle's b and x, for the passes to read from shared memory (every
// thread of the block calls it: it ends with a block barrier)
template <class T>
__device__ __forceinline__ void set_lev0(PTab<T> &tb, int bsel, int xsel) {
    if (threadIdx.x == 0) {
        tb.cur0 = tb.w.lev[0];
        tb.cur0.b = tb.w.vec[bsel];
        tb.cur0.x = tb.w.vec[xsel];
    }
    __syncthreads();
}

// ---------------------------------------------------------------- slots
template <class T> struct alignas(2 * sizeof(T)) Two { T a, b; };
template <class T> __device__ __forceinline__ Two<T> ld2(const T *p) { return *reinterpret_cast<const Two<T> *>(p); }
template <class T> __device__ __forceinline__ void st2(T *p, T a, T b) { *reinterpret_cast<Two<T> *>(p) = Two<T>{a, b}; }
__device__ __forceinline__ int fdiv(int n, FastDiv f) {
    return (int)((__umulhi((unsigned)n, f.mul) + (unsigned)n) >> f.sh);
}
// slot of node (i, j, l), colour included
template <class T>
__device__ __forceinline__ int sslot(const SLev<T> &v, int i, int j, int l) {
    return (((i + j + l) & 1) ? v.H : 0) + v.hx * (j + v.Ny * l) + (i >> 1);
}
// values of the other colour as a half sweep reads them: two neighbouring slots of row
// (j, l), or one (whose slot may lie just outside the row: its coupling is then zero)
template <class T>
struct SrcX {
    const T *x;
    __device__ __forceinline__ Two<T> two(int m, int, int) const { return ld2(x + m); }
    __device__ __forceinline__ T one(int m, int, int) const { return x[m]; }
};
// black values with the coarse correction added: x + al pw xc
template <class T>
struct SrcP {
    const T *x, *pw, *xc;
    T al;
    int hx, Ny, cx, cy, cz, cNx, cNy, chx, cH;
    __device__ __forceinline__ SrcP(const SLev<T> &v, const SLev<T> &c, T al_)
        : x(v.x + v.H), pw(v.pw + v.H), xc(c.x), al(al_), hx(v.hx), Ny(v.Ny), cx(v.cx), cy(v.cy), cz(v.cz),
          cNx(c.Nx), cNy(c.Ny), chx(c.hx), cH(c.H) {}
    __device__ __forceinline__ T coarse(int t, int j, int l) const {
        const int J = j >> cy, K = l >> cz;
        const int I = min(cx ? t : 2 * t + ((j + l + 1) & 1), cNx - 1);   // (past the row: a padding slot, weight zero)
        return xc[(((I + J + K) & 1) ? cH : 0) + chx * (J + cNy * K) + (I >> 1)];
    }
    __device__ __forceinline__ Two<T> two(int m, int j, int l) const {
        const Two<T> v = ld2(x + m), p = ld2(pw + m);
        const int t = m - hx * (j + Ny * l);
        return Two<T>{v.a + al * p.a * coarse(t, j, l), v.b + al * p.b * coarse(t + 1, j, l)};
    }
    __device__ __forceinline__ T one(int m, int j, int l) const {
        int t = m - hx * (j + Ny * l);
        t = t < 0 ? 0 : (t > hx - 1 ? hx - 1 : t);
        return x[m] + al * pw[m] * coarse(t, j, l);
    }
};

// sum of a_kj x_j over the neighbours of the slots m, m + 1 of colour c in row (j, l)
template <class T, class S>
__device__ __forceinline__ Two<T> nb_sum(const SLev<T> &v, int c, int m, int j, int l, const S &src) {
    const T *A = v.A + c * v.H + m;
    const int o = (j + l + c) & 1;                          // node i = 2 (slot in row) + o
    int me = o ? m + 2 : m - 1;
    me = me < 0 ? 0 : (me > v.H - 1 ? v.H - 1 : me);
    const bool jm = j > 0, jp = j < v.Ny - 1, lm = l > 0, lp = l < v.Nz - 1;
    const Two<T> axm = ld2(A), axp = ld2(A + v.ap), aym = ld2(A + 2 * v.ap), ayp = ld2(A + 3 * v.ap),
                 azm = ld2(A + 4 * v.ap), azp = ld2(A + 5 * v.ap);
    const Two<T> xc = src.two(m, j, l);
    const T e = src.one(me, j, l);
    const Two<T> ym = src.two(jm ? m - v.hx : m, jm ? j - 1 : j, l), yp = src.two(jp ? m + v.hx : m, jp ? j + 1 : j, l);
    const Two<T> zm = src.two(lm ? m - v.sz : m, j, lm ? l - 1 : l), zp = src.two(lp ? m + v.sz : m, j, lp ? l + 1 : l);
    Two<T> s;
    s.a = axm.a * (o ? xc.a : e) + axp.a * (o ? xc.b : xc.a);
    s.b = axm.b * (o ? xc.b : xc.a) + axp.b * (o ? e : xc.b);
    s.a += aym.a * ym.a; s.b += aym.b * ym.b;
    s.a += ayp.a * yp.a; s.b += ayp.b * yp.b;
    s.a += azm.a * zm.a; s.b += azm.b * zm.b;
    s.a += azp.a * zp.a; s.b += azp.b * zp.b;
    return s;
}

// ---------------------------------------------------------------- passes of a level
// Half sweeps over one colour.  SM_B0: black from the first red values; SM_R: red, solving
// its rows exactly; SM_B: black update with the full residual; SM_RP / SM_BP: the same two
// with the coarse correction added to the black values as they are read.
enum { SM_B0, SM_R, SM_B, SM_RP, SM_BP };
template <class T, int MODE>
__device__ PG_PASS void pg_smooth(const SLev<T> &vr, int tid, int nth, const SLev<T> *clr = nullptr, T al = 0) {
    const SLev<T> v = vr;                                   // register copy of the shared-memory view
    constexpr int c = (MODE == SM_R || MODE == SM_RP) ? 0 : 1;
    const int np = v.H >> 1;
    for (int t = tid; t < np; t += nth) {
        const int row = fdiv(t, v.fr), l = fdiv(row, v.fy), j = row - l * v.Ny, m = 2 * t;
        const int k = c * v.H + m;
        const Two<T> D = ld2(v.D + k), b = ld2(v.b + k);
        if constexpr (MODE == SM_RP) {
            const Two<T> s = nb_sum<T>(v, c, m, j, l, SrcP<T>(v, *clr, al));
            st2(v.x + k, (b.a - s.a) * D.a, (b.b - s.b) * D.b);
        } else {
            const SrcX<T> src{v.x + (1 - c) * v.H};
            if constexpr (MODE == SM_B0 || MODE == SM_R) {
                const Two<T> s = nb_sum<T>(v, c, m, j, l, src);
                st2(v.x + k, (b.a - s.a) * D.a, (b.b - s.b) * D.b);
            } else {
                Two<T> x;
                if constexpr (MODE == SM_BP) x = SrcP<T>(v, *clr, al).two(m, j, l);
                else x = ld2(v.x + k);
                const Two<T> g = ld2(v.G + k);
                const Two<T> s = nb_sum<T>(v, c, m, j, l, src);
                st2(v.x + k, x.a + (b.a - g.a * x.a - s.a) * D.a, x.b + (b.b - g.b * x.b - s.b) * D.b);
            }
        }
    }
}
// black values with the coarse correction added
template <class T>
__device__ PG_PASS void pg_prolong(const SLev<T> &vr, const SLev<T> &cl, T al, int tid, int nth) {
    const SLev<T> v = vr;
    const SrcP<T> src(v, cl, al);
    for (int t = tid; t < (v.H >> 1); t += nth) {
        const int row = fdiv(t, v.fr), l = fdiv(row, v.fy), j = row - l * v.Ny;
        const Two<T> x = src.two(2 * t, j, l);
        st2(v.x + v.H + 2 * t, x.a, x.b);
    }
}
// residual of one black slot m (red rows are exact after a sweep)
template <class T>
__device__ __forceinline__ T black_resid(const SLev<T> &v, int m, int j, int l) {
    const T *A = v.A + v.H + m, *x = v.x;
    const int o = (j + l + 1) & 1;
    int xm = m - 1 + o, xp = m + o;
    xm = xm < 0 ? 0 : xm;
    xp = xp > v.H - 1 ? v.H - 1 : xp;
    const int ym = j > 0 ? m - v.hx : m, yp = j < v.Ny - 1 ? m + v.hx : m;
    const int zm = l > 0 ? m - v.sz : m, zp = l < v.Nz - 1 ? m + v.sz : m;
    T s = A[0] * x[xm] + A[v.ap] * x[xp] + A[2 * v.ap] * x[ym] + A[3 * v.ap] * x[yp] + A[4 * v.ap] * x[zm] +
          A[5 * v.ap] * x[zp];
    return v.b[v.H + m] - v.G[v.H + m] * x[v.H + m] - s;
}
// Weighted residual summed into the 2x2x2 aggregates: a warp takes 8 coarse nodes along x
// times the aggregate's 4 rows (lane = 8 (dj + 2 dl) + node), so the fine reads of 8 lanes
// are contiguous; `pre` also writes the coarse level's first red values D b.
template <class T>
__device__ PG_PASS void pg_restrict(const SLev<T> &fr, const SLev<T> &clr, const T *w, int tid, int nth, bool pre) {
    const SLev<T> f = fr, cl = clr;
    const int lane = tid & 31, sub = lane >> 3, dj = sub & 1, dl = sub >> 1;
    const int ng = cl.n8 * cl.Ny * cl.Nz, nw = nth >> 5;
    for (int g = tid >> 5; g < ng; g += nw) {
        const int row = fdiv(g, cl.f8), K = fdiv(row, cl.fy), J = row - K * cl.Ny;
        const int I = 8 * (g - row * cl.n8) + (lane & 7);
        const int j = f.cy ? 2 * J + dj : J, l = f.cz ? 2 * K + dl : K;
        bool ok = I < cl.Nx && j < f.Ny && l < f.Nz && (f.cy || !dj) && (f.cz || !dl);
        if (!f.cx) ok = ok && ((I + j + l) & 1);
        T r = 0;
        if (ok) {
            const int m = (f.cx ? I : I >> 1) + f.hx * (j + f.Ny * l);
            r = black_resid<T>(f, m, j, l);
            if (w) r *= w[f.H + m];
        }
        r += __shfl_xor_sync(0xffffffffu, r, 8);
        r += __shfl_xor_sync(0xffffffffu, r, 16);
        if (sub == 0 && I < cl.Nx) {
            const int q = sslot(cl, I, J, K);
            cl.b[q] = r;
            if (pre && !((I + J + K) & 1)) cl.x[q] = cl.D[q] * r;
        }
    }
}

#define PG_SYNC()                   \
    do {                            \
        if (!pg_sync(s)) return false; \
    } while (0)

// The passes of one level on the way down (pre-smoothing from zero, residual restricted to
// the next level) and on the way up (prolongation, post-smoothing), each pass followed by
// `sync` - the grid barrier, a cluster's, or a barrier of some warps of block 0.
template <class T, class Sync>
__device__ __forceinline__ bool pg_level_down(int tid, int nth, const SLev<T> &v, const SLev<T> &cl, bool twice,
                                              const T *w, bool pre, Sync sync) {
    pg_smooth<T, SM_B0>(v, tid, nth);
    if (!sync()) return false;
    pg_smooth<T, SM_R>(v, tid, nth);
    if (!sync()) return false;
    if (twice) {
        pg_smooth<T, SM_B>(v, tid, nth);
        if (!sync()) return false;
        pg_smooth<T, SM_R>(v, tid, nth);
        if (!sync()) return false;
    }
    pg_restrict<T>(v, cl, w, tid, nth, pre);
    return sync();
}
template <class T, bool FUSED, class Sync>
__device__ __forceinline__ bool pg_level_up(int tid, int nth, const SLev<T> &v, const SLev<T> &cl, bool twice, T al,
                                            Sync sync) {
    if constexpr (FUSED) {
        pg_smooth<T, SM_RP>(v, tid, nth, &cl, al);
        if (!sync()) return false;
        pg_smooth<T, SM_BP>(v, tid, nth, &cl, al);
        if (!sync()) return false;
        pg_smooth<T, SM_R>(v, tid, nth);
        if (!sync()) return false;
    } else {                         // a barrier among a few warps costs less than gathering through the weights
        pg_prolong<T>(v, cl, al, tid, nth);
        if (!sync()) return false;
        for (int q = 0; q < 2; q++) {
            pg_smooth<T, SM_R>(v, tid, nth);
            if (!sync()) return false;
            if (q) break;
            pg_smooth<T, SM_B>(v, tid, nth);
            if (!sync()) return false;
        }
    }
    if (twice) {
        pg_smooth<T, SM_B>(v, tid, nth);
        if (!sync()) return false;
        pg_smooth<T, SM_R>(v, tid, nth);
        if (!sync()) return false;
    }
    return true;
}

// barrier of the first n threads of the block (whole warps), one hardware barrier per level
__device__ __forceinline__ bool warps_sync(int id, int n) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
    return true;
}
// The levels Ls .. coarsest of a V-cycle in block 0's shared memory.  Level L runs on its
// first nt threads (as many as it has pairs of slots; fewer on the deeper levels): the other
// warps wait at the barrier of the level above.  1024-thread barriers and the natural-order
// loops took 15 us a cycle on 1200 + 160 + 24 unknowns, this 8 us.
template <class T>
__device__ __noinline__ void blk_cycle(const PTab<T> &tb, int Ls, int nl, T al, int deep) {
    const SLev<T> *sv = tb.sv;
    const int tid = threadIdx.x;
    int L = Ls;
    for (; L < nl - 1; L++) {
        const int nt = sv[L - Ls].nt;
        if (tid >= nt) break;
        pg_level_down<T>(tid, nt, sv[L - Ls], sv[L + 1 - Ls], L < deep, nullptr, L + 1 < nl - 1,
                         [&]() { return warps_sync(1 + L - Ls, nt); });
    }
    if (L == nl - 1) {                            // coarsest level: x = inverse b, 8 lanes per row
        const SLev<T> &v = sv[nl - 1 - Ls];
        const int n = v.N, q0 = tid & 7;
        const int *slot = tb.slot, *cslot = tb.cslot;
        if (tid < v.nt) {
            for (int r = tid >> 3; r < ((n + 3) & ~3); r += v.nt >> 3) {
                T sum = 0;
                if (r < n) {
#pragma unroll 4
                    for (int q = q0; q < n; q += 8) sum += v.D[r * n + q] * v.b[cslot[q]];
                }
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                sum += __shfl_xor_sync(0xffffffffu, sum, 4);
                if (q0 == 0 && r < n) v.x[slot[r]] = sum;
            }
        }
    }
    // each level's threads meet again: the ones that stopped above it, and those that come up
    for (L = (L == nl - 1 ? nl - 2 : L); L >= Ls; L--) {
        const int nt = sv[L - Ls].nt;
        if (tid >= nt) continue;
        warps_sync(1 + L - Ls, nt);
        pg_level_up<T, false>(tid, nt, sv[L - Ls], sv[L + 1 - Ls], L < deep, al, [&]() { return warps_sync(1 + L - Ls, nt); });
    }
}

// one V(1,1) cycle x = M^-1 b on the level-0 vectors (bsel -> xsel; the first red values D b
// already in x).  Levels 0 .. Lc-1: the whole grid, grid barriers; levels Lc .. Ls-1: the first
// cluster alone, cluster barriers; levels Ls ..: block 0 in shared memory.
template <class T>
__device__ __noinline__ bool pg_vcycle(PS &s, const PArgs &a, PTab<T> &tb, int nl, int bsel, int xsel, int wsel) {
    const int Ls = a.Ls, Lc = (a.csz && !a.onecl) ? a.Lc : Ls;
    const T al = (T)a.alpha;
    const int deep = a.sweeps2 ? a.deep : 0;
    set_lev0<T>(tb, bsel, xsel);
    auto gsync = [&]() { return pg_sync(s); };
    auto lev = [&](int L) -> const SLev<T> & { return L ? tb.w.lev[L] : tb.cur0; };
    auto wt = [&](int L) -> const T * { return (L == 0 && wsel) ? tb.w.w0 : nullptr; };
    for (int L = 0; L < Lc; L++)
        if (!pg_level_down<T>(s.tid, s.nth, lev(L), lev(L + 1), L < deep, wt(L), L + 1 < Ls, gsync)) return false;
    if ((int)blockIdx.x < (Lc < Ls ? a.csz : 1)) {         // the first cluster (or block 0 alone)
        const int tid = blockIdx.x * blockDim.x + threadIdx.x;   // a 1-D grid: the first cluster is blocks 0 .. csz-1
        const int nth = (Lc < Ls ? a.csz : 1) * blockDim.x;
        auto csync = [&]() {
            if (Lc < Ls) cooperative_groups::this_cluster().sync();
            else __syncthreads();
            return true;
        };
        for (int L = Lc; L < Ls; L++)
            pg_level_down<T>(tid, nth, lev(L), lev(L + 1), L < deep, wt(L), L + 1 < Ls, csync);
        if (blockIdx.x == 0) {
            const SLev<T> &g = tb.w.lev[Ls];
            const SLev<T> v = tb.sv[0];
            const int n = 2 * v.H;
            for (int q = threadIdx.x; q < n; q += blockDim.x) {
                const T b = g.b[q];
                v.b[q] = b;
                if (!v.last && q < v.H) v.x[q] = v.D[q] * b;   // (the coarsest level's D is its inverse)
            }
            __syncthreads();
            blk_cycle<T>(tb, Ls, nl, al, deep);
            __syncthreads();
            for (int q = threadIdx.x; q < n; q += blockDim.x) g.x[q] = v.x[q];
        }
        csync();
        for (int L = Ls - 1; L >= Lc; L--) pg_level_up<T, true>(tid, nth, lev(L), lev(L + 1), L < deep, al, csync);
    }
    if (!pg_sync(s)) return false;
    for (int L = Lc - 1; L >= 0; L--)
        if (!pg_level_up<T, true>(s.tid, s.nth, lev(L), lev(L + 1), L < deep, al, gsync)) return false;
    if (blockIdx.x == 0 && threadIdx.x == 0) s.g->vcycles++;
    return true;
}

// ---------------------------------------------------------------- Krylov loops
// y = A x on the black rows, x a preconditioner's result (its red rows give A x = b)
template <class T>
__device__ __forceinline__ Two<T> black_apply(const SLev<T> &v, const T *x, int t) {
    const int row = fdiv(t, v.fr), l = fdiv(row, v.fy), j = row - l * v.Ny, m = 2 * t;
    const Two<T> g = ld2(v.G + v.H + m), xk = ld2(x + v.H + m);
    const Two<T> s = nb_sum<T>(v, 1, m, j, l, SrcX<T>{x});
    return Two<T>{g.a * xk.a + s.a, g.b * xk.b + s.b};
}

// BiCGSTAB iterations (semiconductor_3d.c:2281-2316) on the records `sk` of precision T
// while it is active, from r = rh = p with the first red values D p in ph (d holds
// nothing yet: the first update writes it).  v and t exist on black slots only: on red rows
// A ph = p and A sh = s.
template <class T>
__device__ bool pg_bicg(PS &s, const PArgs &a, PTab<T> &tb, int nl, KrylovS &sk) {
    T *r = tb.w.vec[0], *rh = tb.w.vec[1], *p = tb.w.vec[2], *v = tb.w.vec[3];
    T *ph = tb.w.vec[4], *sh = tb.w.vec[5], *t = tb.w.vec[6], *d = tb.w.vec[7];
    const int H = tb.w.lev[0].H, np = H >> 1;               // pairs of slots per colour
    const T *Dr = tb.w.lev[0].D;
    bool first = true;
    // (thread 0 decides on the next iteration before the block barrier ahead of the loop's test, not
    // after the test: a warp late at it would read the later decision and leave a barrier early)
    if (threadIdx.x == 0) bicg_next(sk);
    __syncthreads();
    while (sk.active) {
        double acc[3], a1[1], a2[2];
        if (sk.pad0) {
            for (int q = s.tid; q < 2 * np; q += s.nth) {
                const int m = 2 * q;
                const Two<T> rk = ld2(r + m);
                st2(rh + m, rk.a, rk.b);
                st2(p + m, rk.a, rk.b);
                if (m < H) { const Two<T> D = ld2(Dr + m); st2(ph + m, D.a * rk.a, D.b * rk.b); }
            }
            PG_SYNC();
        }
        if (!pg_vcycle<T>(s, a, tb, nl, 2, 4, 1)) return false;          // ph = M p
        {
            const SLev<T> l0 = tb.w.lev[0];
            a1[0] = 0.0;
            for (int q = s.tid; q < np; q += s.nth) {
                const int m = 2 * q;
                const Two<T> y = black_apply<T>(l0, ph, q), hb = ld2(rh + H + m), hr = ld2(rh + m), pr = ld2(p + m);
                st2(v + H + m, y.a, y.b);
                a1[0] += (double)hb.a * (double)y.a + (double)hb.b * (double)y.b + (double)hr.a * (double)pr.a +
                         (double)hr.b * (double)pr.b;
            }
        }
        if (!pg_sum<1>(s, a1)) return false;
        if (threadIdx.x == 0) {
            if (fabs(a1[0]) < 1e-300) { sk.active = 0; sk.status = 2; }
            else { sk.rv = a1[0]; sk.al = sk.rho1 / a1[0]; }
        }
        __syncthreads();
        if (!sk.active) break;
        const T al = (T)sk.al;
        a2[0] = a2[1] = 0.0;
        for (int q = s.tid; q < 2 * np; q += s.nth) {       // s = r - al v; rh.s; D s
            const int m = 2 * q;
            const Two<T> rk = ld2(r + m), vk = ld2((m < H ? p : v) + m), h = ld2(rh + m);
            const T x = rk.a - al * vk.a, y = rk.b - al * vk.b;
            st2(r + m, x, y);
            if (m < H) { const Two<T> D = ld2(Dr + m); st2(sh + m, D.a * x, D.b * y); }
            a2[0] += (double)x * (double)x + (double)y * (double)y;
            a2[1] += (double)h.a * (double)x + (double)h.b * (double)y;
        }
        if (!pg_sum<2>(s, a2)) return false;
        const double rhs_ = a2[1];
        if (threadIdx.x == 0) {
            sk.ss = a2[0];
            if (sqrt(a2[0]) <= sk.tgt) { sk.half = 1; sk.rr = a2[0]; }
        }
        __syncthreads();
        if (sk.half) {                                      // half-step exit: d += al ph
            for (int q = s.tid; q < 2 * np; q += s.nth) {
                const int m = 2 * q;
                const Two<T> x = ld2(ph + m);
                Two<T> y{0, 0};
                if (!first) y = ld2(d + m);
                st2(d + m, y.a + al * x.a, y.b + al * x.b);
            }
            if (threadIdx.x == 0) { sk.active = 0; sk.status = 1; }
            PG_SYNC();
            return true;
        }
        if (!pg_vcycle<T>(s, a, tb, nl, 0, 5, 1)) return false;          // sh = M s
        {
            const SLev<T> l0 = tb.w.lev[0];
            acc[0] = acc[1] = acc[2] = 0.0;
            for (int q = s.tid; q < np; q += s.nth) {
                const int m = 2 * q;
                const Two<T> y = black_apply<T>(l0, sh, q), rb = ld2(r + H + m), rr = ld2(r + m);
                const Two<T> hb = ld2(rh + H + m), hr = ld2(rh + m);
                st2(t + H + m, y.a, y.b);
                const double rs = (double)rr.a * (double)rr.a + (double)rr.b * (double)rr.b;
                acc[0] += (double)y.a * (double)y.a + (double)y.b * (double)y.b + rs;
                acc[1] += (double)y.a * (double)rb.a + (double)y.b * (double)rb.b + rs;
                acc[2] += (double)hb.a * (double)y.a + (double)hb.b * (double)y.b + (double)hr.a * (double)rr.a +
                          (double)hr.b * (double)rr.b;
            }
        }
        if (!pg_sum<3>(s, acc)) return false;
        if (threadIdx.x == 0) {
            sk.tt = acc[0]; sk.ts = acc[1];
            sk.om = acc[0] > 0.0 ? acc[1] / acc[0] : 0.0;
            const double rho = rhs_ - sk.om * acc[2];        // rh . (s - om t)
            sk.be = sk.om != 0.0 ? (rho / sk.rho1) * (sk.al / sk.om) : 0.0;
            sk.rho1 = rho;
        }
        __syncthreads();
        a1[0] = 0.0;
        {
            const T om = (T)sk.om, be = (T)sk.be;
            for (int q = s.tid; q < 2 * np; q += s.nth) {
                const int m = 2 * q;
                const bool red = m < H;
                const Two<T> rk = ld2(r + m), pk = ld2(p + m), x = ld2(ph + m), z = ld2(sh + m);
                const Two<T> vk = red ? pk : ld2(v + m), tk = red ? rk : ld2(t + m);
                Two<T> y{0, 0};
                if (!first) y = ld2(d + m);
                st2(d + m, y.a + (al * x.a + om * z.a), y.b + (al * x.b + om * z.b));
                const T ra = rk.a - om * tk.a, rb = rk.b - om * tk.b;
                const T pa = ra + be * (pk.a - om * vk.a), pb = rb + be * (pk.b - om * vk.b);
                st2(r + m, ra, rb);
                st2(p + m, pa, pb);
                if (red) { const Two<T> D = ld2(Dr + m); st2(ph + m, D.a * pa, D.b * pb); }
                a1[0] += (double)ra * (double)ra + (double)rb * (double)rb;
            }
        }
        first = false;
        if (!pg_sum<1>(s, a1)) return false;
        if (threadIdx.x == 0) {
            sk.rr = a1[0];
            const double rn = sqrt(a1[0]);
            if (rn <= sk.tgt || sk.om == 0.0) { sk.active = 0; sk.status = 1; }
            else {
                if (rn < 0.99 * sk.rbest) { sk.rbest = rn; sk.stall = 0; }
                else if (++sk.stall > 40) { sk.active = 0; sk.status = 2; }
            }
            bicg_next(sk);
        }
        __syncthreads();
    }
    if (first) {                                            // nothing was added: d = 0
        for (int q = s.tid; q < 2 * np; q += s.nth) st2(d + 2 * q, T(0), T(0));
        PG_SYNC();
    }
    return true;
}

// PCG iterations (semiconductor_3d.c:2194-2206) from r with the first red values D r in z:
// one reduction per iteration for rz = r.z and z.A z, the step length from
// p.A p = z.A z - be^2 (p.A p of the last iteration) and A p by the recurrence A z + be A p.
template <class T>
__device__ bool pg_pcg(PS &s, const PArgs &a, PTab<T> &tb, int nl, KrylovS &sk) {
    T *r = tb.w.vec[0], *z = tb.w.vec[1], *p = tb.w.vec[2], *q = tb.w.vec[3], *w = tb.w.vec[4], *d = tb.w.vec[7];
    const int H = tb.w.lev[0].H, np = H >> 1;
    const T *Dr = tb.w.lev[0].D;
    bool first = true;
    for (;;) {
        if (!pg_vcycle<T>(s, a, tb, nl, 0, 1, 0)) return false;          // z = M r
        double acc[2] = {0.0, 0.0};
        {
            const SLev<T> l0 = tb.w.lev[0];
            for (int u = s.tid; u < np; u += s.nth) {       // on red rows A z = r
                const int m = 2 * u;
                const Two<T> y = black_apply<T>(l0, z, u), zb = ld2(z + H + m), zr = ld2(z + m), rb = ld2(r + H + m),
                             rr = ld2(r + m);
                st2(w + H + m, y.a, y.b);
                const double red = (double)rr.a * (double)zr.a + (double)rr.b * (double)zr.b;
                acc[0] += (double)rb.a * (double)zb.a + (double)rb.b * (double)zb.b + red;
                acc[1] += (double)zb.a * (double)y.a + (double)zb.b * (double)y.b + red;
            }
        }
        if (!pg_sum<2>(s, acc)) return false;
        if (threadIdx.x == 0) {
            const double rz = acc[0];
            sk.be = 0.0;
            if (first) {
                sk.rz0 = rz;
                sk.it = 0;
                sk.status = rz > 0.0 ? 0 : 2;
                sk.active = rz > 0.0;
                sk.pq = acc[1];
            } else if (!(rz > sk.rtol * sk.rtol * sk.rz0)) { sk.active = 0; sk.status = 1; }
            else if (sk.it >= sk.maxit) { sk.active = 0; sk.status = 3; }
            else {
                sk.be = rz / sk.rz;
                sk.pq = acc[1] - sk.be * sk.be * sk.pq;
            }
            if (sk.active) {
                sk.rz = rz;
                sk.it++;
                if (!(sk.pq > 0.0)) { sk.active = 0; sk.status = 2; sk.al = 0.0; }
                else sk.al = rz / sk.pq;
            }
        }
        __syncthreads();
        if (!sk.active) break;
        const T al = (T)sk.al, be = (T)sk.be;
        for (int u = s.tid; u < 2 * np; u += s.nth) {
            const int m = 2 * u;
            const bool red = m < H;
            const Two<T> zk = ld2(z + m), rk = ld2(r + m), wk = red ? rk : ld2(w + m);
            Two<T> pk = zk, qk = wk, y{0, 0};
            if (!first) {
                const Two<T> po = ld2(p + m), qo = ld2(q + m);
                pk = Two<T>{zk.a + be * po.a, zk.b + be * po.b};
                qk = Two<T>{wk.a + be * qo.a, wk.b + be * qo.b};
                y = ld2(d + m);
            }
            st2(p + m, pk.a, pk.b);
            st2(q + m, qk.a, qk.b);
            st2(d + m, y.a + al * pk.a, y.b + al * pk.b);
            const T ra = rk.a - al * qk.a, rb = rk.b - al * qk.b;
            st2(r + m, ra, rb);
            if (red) { const Two<T> D = ld2(Dr + m); st2(z + m, D.a * ra, D.b * rb); }
        }
        first = false;
        PG_SYNC();
    }
    if (first) {
        for (int u = s.tid; u < 2 * np; u += s.nth) st2(d + 2 * u, T(0), T(0));
        PG_SYNC();
    }
    return true;
}

// ---------------------------------------------------------------- set-up
// nodes (2t, j, l) and (2t + 1, j, l) of slot u = t + hx row: both colours of one slot
struct Pair { int t, j, l, row; };
template <class T>
__device__ __forceinline__ Pair slot_row(const SLev<T> &v, int u) {
    Pair p;
    p.row = fdiv(u >> 1, v.fr);
    p.t = u - p.row * v.hx;
    p.l = fdiv(p.row, v.fy);
    p.j = p.row - p.l * v.Ny;
    return p;
}
// sum_j a_kj x_j of the natural-order FP64 row k and, in fl, sum_j |a_kj x_j|; a[] keeps the row
// Couplings that leave the domain are taken as zero and their neighbour is the node itself, so
// every load is unconditional (loads behind branches are waited for one by one)
template <class F>
__device__ __forceinline__ double row64(const double *A, int ap, int k, int i, int j, int l, int Nx, int Ny, int Nz,
                                        double (&a)[7], F x, double &fl) {
    const int NxNy = Nx * Ny;
    const bool e[6] = {i > 0, i < Nx - 1, j > 0, j < Ny - 1, l > 0, l < Nz - 1};
    double y[7];
#pragma unroll
    for (int q = 0; q < 7; q++) a[q] = A[q * ap + k];
    y[0] = x(k, i, j, l);
    y[1] = x(e[0] ? k - 1 : k, e[0] ? i - 1 : i, j, l);
    y[2] = x(e[1] ? k + 1 : k, e[1] ? i + 1 : i, j, l);
    y[3] = x(e[2] ? k - Nx : k, i, e[2] ? j - 1 : j, l);
    y[4] = x(e[3] ? k + Nx : k, i, e[3] ? j + 1 : j, l);
    y[5] = x(e[4] ? k - NxNy : k, i, j, e[4] ? l - 1 : l);
    y[6] = x(e[5] ? k + NxNy : k, i, j, e[5] ? l + 1 : l);
    double t = a[0] * y[0], sum = t;
    fl = fabs(t);
#pragma unroll
    for (int q = 1; q < 7; q++) {
        if (!e[q - 1]) a[q] = 0.0;
        t = a[q] * y[q];
        sum += t;
        fl += fabs(t);
    }
    return sum;
}
// The level-0 system of the launch: r = b - A x with the FP64 operator (its squared norm and
// the squared rounding floor sum_k (sum_j |a_kj x_j| + |b_k|)^2 in acc,
// semiconductor_3d.c:2244-2268), and the colour-ordered copy of the operator, the row weights
// and r (rh = p = r) in precision T; padding slots are zeroed.  FP32 PCG starts from x = 0.
template <class T, int KIND>
__device__ __forceinline__ void pg_load(const DevP &P, const PTab<T> &tb, const PS &s, double (&acc)[2]) {
    const SLev<T> v = tb.w.lev[0];
    constexpr bool zero_x = KIND == PK_PCG && std::is_same<T, float>::value;
    const double *x = P.sol;
    for (int u = s.tid; u < v.H; u += s.nth) {
        const Pair p = slot_row(v, u);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int i = 2 * p.t + q, m = (((i + p.j + p.l) & 1) ? v.H : 0) + u;
            double a[7] = {0, 0, 0, 0, 0, 0, 0}, rk = 0.0, w = 0.0;
            if (i < v.Nx) {
                const int k = i + v.Nx * p.row;
                double fl;
                const double b = P.rhs[k];
                const double sum = row64(tb.A64, tb.ap64, k, i, p.j, p.l, v.Nx, v.Ny, v.Nz, a,
                                         [&](int kk, int, int, int) { return zero_x ? 0.0 : x[kk]; }, fl);
                fl += fabs(b);
                rk = b - sum;
                acc[0] += rk * rk;
                acc[1] += fl * fl;
                if (KIND == PK_REFINED) P.wk[0][k] = rk;
                if (KIND != PK_PCG) w = P.dsc[k];
            }
            const T g = (T)a[0];
            v.G[m] = g;
            if (!((i + p.j + p.l) & 1) && i < v.Nx) v.D[m] = g != T(0) ? T(1) / g : T(1);   // red pivot
#pragma unroll
            for (int e = 0; e < 6; e++) v.A[e * v.ap + m] = (T)a[1 + e];
            tb.w.vec[0][m] = (T)rk;
            if (KIND != PK_PCG) {
                tb.w.vec[1][m] = (T)rk;
                tb.w.vec[2][m] = (T)rk;
                tb.w.w0[m] = (T)w;
            }
            if (i >= v.Nx) { v.pw[m] = 0; v.D[m] = 0; }
        }
    }
}
// reciprocal red-black D-ILU pivots of the black slots, a_kk - sum a_kr a_rk / a_rr, guarded
// as the reference guards its ILU pivots (semiconductor_3d.c:1937-1938); the red ones, 1 / a_rr,
// are written with the operator
template <class T>
__device__ PG_SETUP void pg_pivots(const SLev<T> &vr, int tid, int nth) {
    const SLev<T> v = vr;
    for (int u = tid; u < v.H; u += nth) {
        const Pair p = slot_row(v, u);
        const int o = (p.j + p.l + 1) & 1, i = 2 * p.t + o, m = v.H + u;
        const bool ok[6] = {i > 0, i < v.Nx - 1, p.j > 0, p.j < v.Ny - 1, p.l > 0, p.l < v.Nz - 1};
        const int nbr[6] = {u - 1 + o, u + o, u - v.hx, u + v.hx, u - v.sz, u + v.sz};
        const T *A = v.A + m, *R = v.A;
        const T g = v.G[m];
        T sum = 0;
#pragma unroll
        for (int e = 0; e < 6; e++) {
            const int n = ok[e] ? nbr[e] : u;
            const T c = A[e * v.ap] * R[(e ^ 1) * v.ap + n] * v.D[n];
            sum += ok[e] ? c : T(0);
        }
        T d = g - sum;
        if (!(d > T(1e-8) * fabs(g))) d = g;
        if (!(d != T(0))) d = 1;
        v.D[m] = i < v.Nx ? T(1) / d : T(0);
    }
}
// Slotboom weights of the level's nodes towards the next one, and that level's reference
// potentials (semiconductor_3d.c:2092-2117); thread per coarse node.  phf / phc: the levels'
// reference potentials in natural order (phf null: level 0, from the state)
template <class T>
__device__ PG_SETUP void pg_weights(const DevP &P, const SLev<T> &f, const SLev<T> &cl, const double *phf,
                                           double *phc, int qsign, int tid, int nth) {
    for (int K = tid; K < cl.N; K += nth) {
        const Node c = unidx(K, cl.Nx, cl.Ny);
        const Agg g = agg_range(f, c.i, c.j, c.l);
        double p[8], mx = PH_NONE;
        if (qsign) {
#pragma unroll
            for (int q = 0; q < 8; q++) {                   // (an aggregate cut short repeats its last nodes)
                const int k = min(g.i0 + (q & 1), g.i1) +
                              f.Nx * (min(g.j0 + ((q >> 1) & 1), g.j1) + f.Ny * min(g.l0 + (q >> 2), g.l1));
                p[q] = phf ? phf[k] : ph0(P, k, qsign);
            }
#pragma unroll
            for (int q = 0; q < 8; q++) mx = fmax(mx, p[q]);
            phc[K] = mx;
        }
#pragma unroll
        for (int q = 0; q < 8; q++) {
            T wt = 1;
            if (qsign) {
                const double e = (p[q] <= 0.5 * PH_NONE) ? -800.0 : p[q] - mx;
                wt = (T)(e < -700.0 ? 0.0 : exp(e));
            }
            f.pw[sslot(f, min(g.i0 + (q & 1), g.i1), min(g.j0 + ((q >> 1) & 1), g.j1), min(g.l0 + (q >> 2), g.l1))] = wt;
        }
    }
}
// Petrov-Galerkin coarse operator P^T W A P (semiconductor_3d.c:2003-2027), summed in FP64:
// lanes as in pg_restrict, each lane the two nodes of one of the aggregate's rows
template <class T>
__device__ PG_SETUP void pg_galerkin(const SLev<T> &fr, const SLev<T> &clr, const T *w, int tid, int nth) {
    const SLev<T> f = fr, cl = clr;
    const int lane = tid & 31, sub = lane >> 3, dj = sub & 1, dl = sub >> 1;
    const int ng = cl.n8 * cl.Ny * cl.Nz, nw = nth >> 5;
    for (int g = tid >> 5; g < ng; g += nw) {
        const int row = fdiv(g, cl.f8), K = fdiv(row, cl.fy), J = row - K * cl.Ny;
        const int I = 8 * (g - row * cl.n8) + (lane & 7);
        const int j = f.cy ? 2 * J + dj : J, l = f.cz ? 2 * K + dl : K;
        const bool ok = I < cl.Nx && j < f.Ny && l < f.Nz && (f.cy || !dj) && (f.cz || !dl);
        double a[7] = {0, 0, 0, 0, 0, 0, 0};
        if (ok) {
            const int i0 = f.cx ? 2 * I : I, i1 = f.cx ? min(2 * I + 1, f.Nx - 1) : I;
            const int j0 = f.cy ? 2 * J : J, j1 = f.cy ? min(2 * J + 1, f.Ny - 1) : J;
            const int l0 = f.cz ? 2 * K : K, l1 = f.cz ? min(2 * K + 1, f.Nz - 1) : K;
            const bool ej0 = j > 0, ej1 = j < f.Ny - 1, el0 = l > 0, el1 = l < f.Nz - 1;
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int i = i0 + q;
                const bool in = i <= i1;
                const int ii = in ? i : i0, m = sslot(f, ii, j, l);
                const T *A = f.A + m;
                const double wk = in ? (w ? (double)w[m] : 1.0) : 0.0;
                // (a coupling that leaves the domain is zero: any weight will do)
                const T g0 = f.G[m], p0 = f.pw[m];
                const T am[6] = {A[0], A[f.ap], A[2 * f.ap], A[3 * f.ap], A[4 * f.ap], A[5 * f.ap]};
                const T pn[6] = {f.pw[sslot(f, max(ii - 1, 0), j, l)], f.pw[sslot(f, min(ii + 1, f.Nx - 1), j, l)],
                                 f.pw[sslot(f, ii, ej0 ? j - 1 : j, l)], f.pw[sslot(f, ii, ej1 ? j + 1 : j, l)],
                                 f.pw[sslot(f, ii, j, el0 ? l - 1 : l)], f.pw[sslot(f, ii, j, el1 ? l + 1 : l)]};
                const bool inner[6] = {ii - 1 >= i0, ii + 1 <= i1, j - 1 >= j0, j + 1 <= j1, l - 1 >= l0, l + 1 <= l1};
                a[0] += wk * (double)g0 * (double)p0;
#pragma unroll
                for (int e = 0; e < 6; e++) {
                    const double c = wk * (double)am[e] * (double)pn[e];
                    a[0] += inner[e] ? c : 0.0;
                    a[1 + e] += inner[e] ? 0.0 : c;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 7; q++) {
            a[q] += __shfl_xor_sync(0xffffffffu, a[q], 8);
            a[q] += __shfl_xor_sync(0xffffffffu, a[q], 16);
        }
        if (sub == 0 && I < 2 * cl.hx) {                    // (padding slots: zeros, a[] is zero there)
            const int q = sslot(cl, I, J, K);
            if (I >= cl.Nx) {
                if (!cl.last) cl.pw[q] = 0;
                cl.x[q] = 0;
                cl.b[q] = 0;
            } else if (a[0] == 0. && a[1] == 0. && a[2] == 0. && a[3] == 0. && a[4] == 0. && a[5] == 0. && a[6] == 0.) a[0] = 1.;
            const T g = (T)a[0];
            cl.G[q] = g;
            if (!cl.last && !((I + J + K) & 1))              // red pivot (0 in a padding slot)
                cl.D[q] = I >= cl.Nx ? T(0) : (g != T(0) ? T(1) / g : T(1));
#pragma unroll
            for (int e = 0; e < 6; e++) cl.A[e * cl.ap + q] = (T)a[1 + e];
        }
    }
}
// Dense inverse of the coarsest level (n <= 64) by Gauss-Jordan with partial pivoting in FP64
// (tiny pivots guarded as semiconductor_3d.c:2066 does).  A chain of n dependent steps, so what
// counts is the length of one: two or four warps only (warp w: rows 32 (w / 2) + lane, the
// columns of parity w & 1, NC of them in registers), rows are never moved and stay unscaled
// until the end (row piv[c] plays row c), and the columns turn by one register when their
// parity's pivot is done, so that the pivot column is always a[0] and no step selects by the
// column's number.  Per step the warps exchange the column and the pivot row through shared
// memory (two barriers of those warps).  D[c n + q] is left as element (c, piv[q]) of the
// inverse.  24 unknowns 10 us, 60 unknowns 22 us; 8 lanes per row of all 16 warps took 16 and
// 50 us.
template <class T, int NC>
__device__ __noinline__ void invert_rows(T *D, int n, int nt, int *piv) {
    __shared__ double col[2][COARSE_MAX];
    __shared__ __align__(16) double prow[2][2][COARSE_MAX / 2];
    const int tid = threadIdx.x, lane = tid & 31, ch = (tid >> 5) & 1, r = 32 * (tid >> 6) + lane;
    const bool row = r < n;
    double a[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) a[i] = row && 2 * i + ch < n ? (double)D[r * n + 2 * i + ch] : 0.0;
    bool open0 = lane < n, open1 = lane + 32 < n;            // rows lane and lane + 32 not used yet
    int mine = 0;                                            // the column this row was the pivot of
    double scale = 0.0;                                      // and its reciprocal pivot
    for (int c = 0; c < n; c++) {
        double *cc = col[c & 1];
        const bool own = ch == (c & 1);
        if (own) cc[r] = a[0];                               // (rows past n: zeros)
        warps_sync(1, nt);
        unsigned key = 0;                                    // |a| to 15 bits of mantissa, ties to the lower row
        {
            const unsigned h0 = (unsigned)__double2hiint(cc[lane]), k0 = ((h0 << 1) & ~63u) | (unsigned)(63 - lane);
            key = open0 ? k0 : 0u;
            if (NC > 16) {
                const unsigned h1 = (unsigned)__double2hiint(cc[lane + 32]), k1 = ((h1 << 1) & ~63u) | (unsigned)(31 - lane);
                key = max(key, open1 ? k1 : 0u);
            }
        }
        const double f = cc[r];
        const int p = 63 - (int)(__reduce_max_sync(0xffffffffu, key) & 63u);
        const double d = cc[p], inv = 1.0 / (fabs(d) > 1e-300 ? d : 1e-300);
        open0 = open0 && p != lane;
        open1 = open1 && p != lane + 32;
        double2 *pw = reinterpret_cast<double2 *>(prow[c & 1][ch]);
        if (r == p) {
            mine = c;
            scale = inv;
            if (own) piv[c] = p;
#pragma unroll
            for (int i = 0; i < NC / 2; i++) pw[i] = make_double2(a[2 * i], a[2 * i + 1]);
        }
        const double g = r == p ? 0.0 : -f * inv;
        warps_sync(1, nt);
        if (own) {
#pragma unroll
            for (int i = 0; i < NC / 2; i++) {
                const double2 q = pw[i];
                if (i) a[2 * i - 1] = a[2 * i] + g * q.x;
                a[2 * i] = a[2 * i + 1] + g * q.y;
            }
            a[NC - 1] = r == p ? 1.0 : g;
        } else {
#pragma unroll
            for (int i = 0; i < NC / 2; i++) {
                const double2 q = pw[i];
                a[2 * i] += g * q.x;
                a[2 * i + 1] += g * q.y;
            }
        }
    }
    const int k = (n + 1 - ch) >> 1;                         // columns of this parity: the turns made
    T *out = D + mine * n + ch + 2 * k;
    if (row)
#pragma unroll
        for (int i = 0; i < NC; i++) {
            if (i + k >= NC) out[2 * (i - NC)] = (T)(a[i] * scale);   // slots below k: 2 (i + k - NC) + ch
        }
}
// the coarsest level's matrix spread out in v.D (zero before), then its inverse
template <class T>
__device__ __forceinline__ void blk_invert(PTab<T> &tb, const SLev<T> &v) {
    __shared__ int piv[COARSE_MAX];
    const int n = v.N, tid = threadIdx.x, nt = n > 32 ? 128 : 64;
    if (tid < nt) {
        int m = 0;
        if (tid < n) {
            const Node c = unidx(tid, v.Nx, v.Ny);
            const int NxNy = v.Nx * v.Ny;
            m = sslot(v, c.i, c.j, c.l);
            const T *A = v.A + m;
            T *row = v.D + tid * n + tid;
            row[0] = v.G[m];
            if (c.i > 0) row[-1] = A[0];
            if (c.i < v.Nx - 1) row[1] = A[v.ap];
            if (c.j > 0) row[-v.Nx] = A[2 * v.ap];
            if (c.j < v.Ny - 1) row[v.Nx] = A[3 * v.ap];
            if (c.l > 0) row[-NxNy] = A[4 * v.ap];
            if (c.l < v.Nz - 1) row[NxNy] = A[5 * v.ap];
            tb.slot[tid] = m;
        }
        warps_sync(1, nt);
        if (n > 32) invert_rows<T, 32>(v.D, n, nt, piv);
        else invert_rows<T, 16>(v.D, n, nt, piv);
        if (tid < n) tb.cslot[tid] = tb.slot[piv[tid]];
    }
    __syncthreads();
}
// bytes of block 0's shared memory: a level's arrays, and the coarsest level's inverse with
// its scratch
template <class T>
__host__ __device__ inline size_t ssm_level(int H, int ap, int n, bool last) {
    if (last)
        return al16((size_t)6 * ap * sizeof(T)) + 3 * al16((size_t)2 * H * sizeof(T)) + al16((size_t)n * n * sizeof(T));
    return al16((size_t)6 * ap * sizeof(T)) + 5 * al16((size_t)2 * H * sizeof(T));
}
// Views of the levels Ls .. nl-1 in block 0's shared memory, a thread per level, and all of it
// zeroed (padding slots, the coarsest matrix); done while the block waits at the first barrier
template <class T>
__device__ __forceinline__ void ssm_views(PTab<T> &tb, int Ls, int nl, unsigned char *base, int tid, int nth) {
    size_t all = 0;
    for (int L = Ls; L < nl; L++) all += ssm_level<T>(tb.w.lev[L].H, tb.w.lev[L].ap, tb.w.lev[L].N, L == nl - 1);
    for (int q = tid; q < (int)(all / 16); q += nth) reinterpret_cast<int4 *>(base)[q] = make_int4(0, 0, 0, 0);
    const int L = Ls + tid;
    if (L < nl) {
        unsigned char *p = base;
        for (int K = Ls; K < L; K++) p += ssm_level<T>(tb.w.lev[K].H, tb.w.lev[K].ap, tb.w.lev[K].N, false);
        SLev<T> &v = tb.sv[L - Ls];
        v = tb.w.lev[L];
        const size_t nb = al16((size_t)2 * v.H * sizeof(T));
        v.A = reinterpret_cast<T *>(p); p += al16((size_t)6 * v.ap * sizeof(T));
        v.G = reinterpret_cast<T *>(p); p += nb;
        v.D = reinterpret_cast<T *>(p); p += v.last ? al16((size_t)v.N * v.N * sizeof(T)) : nb;
        if (!v.last) { v.pw = reinterpret_cast<T *>(p); p += nb; }
        v.x = reinterpret_cast<T *>(p); p += nb;
        v.b = reinterpret_cast<T *>(p);
        // threads of a level: a pair of slots each, a warp per 8 coarse nodes of its restriction,
        // 8 lanes per row of the dense inverse, and no fewer than the levels below
        int nt = 0;
        for (int K = L; K < nl; K++) {
            const SLev<T> &w = tb.w.lev[K];
            nt = max(nt, w.last ? 8 * w.N : max(w.H >> 1, 32 * tb.w.lev[K + 1].n8 * tb.w.lev[K + 1].Ny * tb.w.lev[K + 1].Nz));
        }
        v.nt = min((nt + 31) & ~31, (int)blockDim.x);
    }
}
// The multigrid set-up of the system loaded by pg_load (the reference's mg_setup,
// semiconductor_3d.c:2126-2148): one grid pass per large level - its pivots, the Galerkin
// operator of the next level and that level's weights - and the small levels in block 0's
// shared memory.  `xr` takes the first red values D r of the solve.
template <class T>
__device__ __noinline__ bool pg_setup(const DevP &P, PS &s, const PArgs &a, PTab<T> &tb, int nl, T *xr) {
    const int Ls = a.Ls, qsign = a.qsign;
    for (int L = 0; L < Ls; L++) {
        const SLev<T> &f = tb.w.lev[L], &cl = tb.w.lev[L + 1];
        pg_galerkin<T>(f, cl, (L == 0 && qsign) ? tb.w.w0 : nullptr, s.tid, s.nth);
        pg_pivots<T>(f, s.tid, s.nth);
        if (L == 0)
            for (int u = s.tid; u < f.H; u += s.nth) xr[u] = f.D[u] * tb.w.vec[0][u];
        if (L + 1 < Ls) pg_weights<T>(P, cl, tb.w.lev[L + 2], PT<T>::lev(P, L + 1).ph, PT<T>::lev(P, L + 2).ph, qsign, s.tid, s.nth);
        PG_SYNC();
    }
    if (blockIdx.x == 0) {
        const int tid = threadIdx.x, nth = blockDim.x;
        {
            const SLev<T> &g = tb.w.lev[Ls], &v = tb.sv[0];
            // the first small level as pg_galerkin left it, padding slots included (the black
            // pivots are stale, pg_pivots writes them below; the coarsest level has none)
            for (int e = 0; e < (v.last ? 2 : 3); e++) {
                const int4 *src = reinterpret_cast<const int4 *>(e == 0 ? g.A : e == 1 ? g.G : g.D);
                int4 *dst = reinterpret_cast<int4 *>(e == 0 ? v.A : e == 1 ? v.G : v.D);
                const int n = (e == 0 ? 6 * v.ap : 2 * v.H) * (int)sizeof(T) / 16;   // (2 H: a multiple of 4)
#pragma unroll 4
                for (int q = tid; q < n; q += nth) dst[q] = src[q];
            }
            __syncthreads();
        }
        for (int L = Ls; L < nl - 1; L++) {
            const SLev<T> &v = tb.sv[L - Ls], &cl = tb.sv[L + 1 - Ls];
            pg_weights<T>(P, v, cl, PT<T>::lev(P, L).ph, PT<T>::lev(P, L + 1).ph, qsign, tid, nth);
            pg_pivots<T>(v, tid, nth);
            __syncthreads();
            pg_galerkin<T>(v, cl, nullptr, tid, nth);
            __syncthreads();
        }
        blk_invert<T>(tb, tb.sv[nl - 1 - Ls]);
    }
    return true;
}

// natural-order sol += d
template <class T>
__device__ __forceinline__ void pg_add_solution(const DevP &P, const PTab<T> &tb, const PS &s, bool assign) {
    const SLev<T> v = tb.w.lev[0];
    const T *d = tb.w.vec[7];
    for (int u = s.tid; u < v.H; u += s.nth) {
        const Pair p = slot_row(v, u);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int i = 2 * p.t + q;
            if (i >= v.Nx) continue;
            const double x = (double)d[(((i + p.j + p.l) & 1) ? v.H : 0) + u];
            double *sol = P.sol + i + v.Nx * p.row;
            *sol = assign ? x : *sol + x;
        }
    }
}

// ---------------------------------------------------------------- the solve kernels
// T: precision of the Krylov iterations and the hierarchy.  PK_PCG: the Poisson Newton
// system from the present sol (T = float: from zero, and the result goes to the FP64 sol
// when it converged).  PK_BICG (T = double): the continuity system from the present sol.
// PK_REFINED (T = float): FP64 refinement steps around FP32 BiCGSTAB.
template <class T, int KIND>
__global__ void __launch_bounds__(PT_TPB, 1) k_persist(const DevP *Ps, PArgs a) {
    const DevP &P = Ps[0];
    extern __shared__ __align__(16) unsigned char sraw[];
    __shared__ PTab<T> tb;
    __shared__ KrylovS sk, so;                    // the loop's record (and the outer one: PK_REFINED)
    PS s;
    s.g = P.pgrid;
    s.target = 0;
    s.rb = 0;
    s.tid = blockIdx.x * blockDim.x + threadIdx.x;
    s.nth = gridDim.x * blockDim.x;
    s.wait_ns = PG_WAIT_NS;
    s.trace = a.trace;
    s.ntrace = a.ntrace;
    s.mode = a.barmode;
    s.onecl = a.onecl;
    const int nl = P.nlev;
    {
        const int *src = reinterpret_cast<const int *>(swork<T>(P));
        int *dst = reinterpret_cast<int *>(&tb.w);
        for (int q = threadIdx.x; q < (int)(sizeof(SWork<T>) / sizeof(int)); q += blockDim.x) dst[q] = src[q];
        if (threadIdx.x == 0) {
            tb.A64 = P.A[0];
            tb.ap64 = (int)(P.A[1] - P.A[0]);
            sk = a.rec[0];
            so = a.rec[1];
        }
    }
    __syncthreads();
    // the system, its first residual and (level 0 -> 1) weights
    double acc[2] = {0.0, 0.0};
    pg_load<T, KIND>(P, tb, s, acc);
    pg_weights<T>(P, tb.w.lev[0], tb.w.lev[1], nullptr, PT<T>::lev(P, 1).ph, a.qsign, s.tid, s.nth);
    if (!pg_sum<2>(s, acc, [&]() { if (blockIdx.x == 0) ssm_views<T>(tb, a.Ls, nl, sraw, threadIdx.x - 32, blockDim.x - 32); })) return;
    if constexpr (KIND != PK_PCG) {
        if (threadIdx.x == 0) {
            KrylovS &rec = KIND == PK_REFINED ? so : sk;
            const double rtol = KIND == PK_REFINED ? so.rtol : a.rtol, atol = KIND == PK_REFINED ? so.atol : a.atol;
            rec.rr = acc[0]; rec.fl = acc[1];
            rec.r0 = sqrt(acc[0]);
            rec.tgt = fmax(rtol * rec.r0, atol * sqrt(acc[1]));
            rec.rbest = rec.r0; rec.stall = 0; rec.it = 0; rec.half = 0; rec.rho1 = acc[0];
            if (!(rec.r0 > rec.tgt)) { rec.active = 0; rec.status = 1; }
            else { rec.active = 1; rec.status = 0; }
        }
        __syncthreads();
    }
    const bool go = KIND == PK_PCG || (KIND == PK_REFINED ? so.active : sk.active) != 0;
    int steps = 0;
    if (go) {
        if (!pg_setup<T>(P, s, a, tb, nl, tb.w.vec[KIND == PK_PCG ? 1 : 4])) return;
        if constexpr (KIND == PK_PCG) {
            if (!pg_pcg<T>(s, a, tb, nl, sk)) return;
            if (std::is_same<T, double>::value || sk.status == 1)
                pg_add_solution<T>(P, tb, s, std::is_same<T, float>::value);
        } else if constexpr (KIND == PK_BICG) {
            if (!pg_bicg<T>(s, a, tb, nl, sk)) return;
            pg_add_solution<T>(P, tb, s, false);
        } else {                                  // PK_REFINED
            double *x = P.sol, *r64 = P.wk[0];
            double r32 = so.rr;                   // squared norm of the FP32 right-hand side (the FP64 one's, rounded)
            for (; steps < a.maxsteps && so.active; steps++) {
                if (threadIdx.x == 0) {
                    sk.rr = r32;
                    sk.r0 = sqrt(r32);
                    sk.tgt = fmax(sk.rtol * sk.r0, sk.atol * so.tgt);
                    sk.rho1 = r32; sk.rbest = sk.r0; sk.stall = 0; sk.it = 0; sk.half = 0;
                    sk.body_runs = 0;
                    sk.maxit = so.maxit - so.it;
                    sk.status = 0;
                    sk.active = (sk.r0 > sk.tgt && sk.maxit > 0) ? 1 : 0;
                }
                __syncthreads();
                if (!pg_bicg<T>(s, a, tb, nl, sk)) return;
                // x += d; r -= A d (FP64 operator); the next inner start r = rh = p = (float) r
                double au[2] = {0.0, 0.0};
                {
                    const SLev<T> v = tb.w.lev[0];
                    const T *d = tb.w.vec[7];
                    for (int u = s.tid; u < v.H; u += s.nth) {
                        const Pair p = slot_row(v, u);
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            const int i = 2 * p.t + q, c = (i + p.j + p.l) & 1, m = (c ? v.H : 0) + u;
                            if (i >= v.Nx) continue;
                            const int k = i + v.Nx * p.row;
                            double fl, row[7];
                            const double sum = row64(tb.A64, tb.ap64, k, i, p.j, p.l, v.Nx, v.Ny, v.Nz, row,
                                                     [&](int, int ii, int jj, int ll) { return (double)d[sslot(v, ii, jj, ll)]; }, fl);
                            x[k] += (double)d[m];
                            const double rk = r64[k] - sum;
                            r64[k] = rk;
                            const T f = (T)rk;
                            tb.w.vec[0][m] = f; tb.w.vec[1][m] = f; tb.w.vec[2][m] = f;
                            if (!c) tb.w.vec[4][m] = v.D[m] * f;
                            au[0] += rk * rk;
                            au[1] += (double)f * (double)f;
                        }
                    }
                }
                if (!pg_sum<2>(s, au)) return;
                r32 = au[1];
                if (threadIdx.x == 0) {
                    so.it += sk.it;
                    so.body_runs++;
                    so.rr = au[0];
                    const double rn = sqrt(au[0]);
                    if (rn <= so.tgt) { so.active = 0; so.status = 1; }
                    else if (!(rn < 0.5 * so.rbest)) { so.active = 0; so.status = 4; }
                    else if (so.it >= so.maxit) { so.active = 0; so.status = 3; }
                    else so.rbest = rn;
                }
                __syncthreads();
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s.g->rec[0] = sk;
        s.g->rec[1] = so;
        s.g->steps = steps;
        s.g->iters = KIND == PK_REFINED ? so.it : sk.it;
    }
}

// Test of the bounded barrier wait: the last block of the launch never arrives, so every
// other block must give up after wait_ns, set the error word and report ok = 0.
__global__ void k_pg_timeout_probe(PGrid *g, unsigned long long wait_ns, int *ok) {
    PS s;
    s.g = g;
    s.target = 0;
    s.rb = 0;
    s.tid = blockIdx.x * blockDim.x + threadIdx.x;
    s.nth = gridDim.x * blockDim.x;
    s.wait_ns = wait_ns;
    s.trace = nullptr;
    s.ntrace = 0;
    s.mode = 1;
    s.onecl = 0;
    if (blockIdx.x == gridDim.x - 1) return;     // never arrives
    const bool r = pg_sync(s);
    if (threadIdx.x == 0) ok[blockIdx.x] = r ? 1 : 0;
}

// ---------------------------------------------------------------- host side
namespace {
struct KInfo {
    const void *fn = nullptr;
    size_t smem = 0;       // dynamic shared memory the attribute allows
    int blocks = 0;        // co-resident blocks at that size
    int clusters[2] = {};  // co-resident clusters of 8 / 16 CTAs at that size (0: no such launch)
};
std::mutex g_pmu;
int g_persist_mode = -1;   // -1 unread, 0 off, 1 on
int g_persist_blocks = 0;  // blocks per launch (0: every SM's worth)
thread_local int t_persist_blocks = 0;  // this host thread's cap (0: none)
bool g_persist_broken = false;
bool g_coop_ok = false;    // the device supports cooperative launches
unsigned long long *g_trace = nullptr;   // armed barrier timeline (test hook): device buffer
int g_trace_n = 0, g_trace_used = 0;     // its barriers; 1 once a launch has filled it
int g_last_blocks = 0;                   // blocks of the last persistent launch
thread_local int t_shape[2];             // blocks and cluster CTAs of this host thread's last one (test hook)
int g_barmode = 1;         // grid-barrier form (SEMISIM_B200_BARMODE; 1 measured faster than 0)
int g_clusters = 1;        // cluster launches: 0 off, 1 where they gain (persist_run), 2 every grid (SEMISIM_B200_CLUSTERS)
int g_csz = 16;            // CTAs per cluster at most (SEMISIM_B200_CSZ: 8 portable, 16 non-portable)
int g_clevel = 1;          // first level the first cluster runs alone (SEMISIM_B200_CLEVEL)
int g_coop = 1;            // cooperative launch attribute (SEMISIM_B200_COOP=0: plain launch of a
                           //   grid within the co-resident capacity)

template <class T, int KIND>
const void *kfn() { return reinterpret_cast<const void *>(&k_persist<T, KIND>); }

// co-resident clusters of csz CTAs of the kernel at `smem` bytes (0: no clusters)
int cluster_occupancy(const void *fn, size_t smem, int csz) {
    if (csz > 8 && cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t q = {};
    q.gridDim = dim3(csz);
    q.blockDim = dim3(PT_TPB);
    q.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = csz; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    q.attrs = at;
    q.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &q) != cudaSuccess) { cudaGetLastError(); return 0; }
    return n;
}
// co-resident blocks of the kernel at `smem` bytes (0 when it cannot launch)
int occupancy(const void *fn, size_t smem) {
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int per = 0, dev = 0, nsm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, PT_TPB, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return per * nsm;
}
}  // namespace

int persist_enabled() {
    std::lock_guard<std::mutex> lk(g_pmu);
    if (g_persist_mode < 0) {
        const char *e = std::getenv("SEMISIM_B200_PERSIST");
        g_persist_mode = (e && std::atoi(e) == 0) ? 0 : 1;
        if (const char *b = std::getenv("SEMISIM_B200_PBLOCKS")) g_persist_blocks = std::atoi(b);
        if (const char *m = std::getenv("SEMISIM_B200_BARMODE")) g_barmode = std::atoi(m) ? 1 : 0;
        if (const char *m = std::getenv("SEMISIM_B200_CLUSTERS")) g_clusters = std::atoi(m) < 0 ? 0 : (std::atoi(m) > 2 ? 2 : std::atoi(m));
        if (const char *m = std::getenv("SEMISIM_B200_CLEVEL")) g_clevel = std::atoi(m) < 1 ? 1 : std::atoi(m);
        if (const char *m = std::getenv("SEMISIM_B200_CSZ")) g_csz = std::atoi(m) == 8 ? 8 : 16;
        if (const char *m = std::getenv("SEMISIM_B200_COOP")) g_coop = std::atoi(m) != 0;
        int dev = 0, coop = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) cudaGetLastError();
        g_coop_ok = coop != 0;
    }
    return g_persist_mode == 1 && g_coop_ok && !g_persist_broken;
}
void persist_set(int mode, int blocks) {
    persist_enabled();
    std::lock_guard<std::mutex> lk(g_pmu);
    if (mode >= 0) g_persist_mode = mode ? 1 : 0;
    if (blocks >= 0) g_persist_blocks = blocks;
}
void persist_note(int blocks, int csz) { t_shape[0] = blocks; t_shape[1] = csz; }
void persist_shape(int *blocks, int *csz) {
    *blocks = t_shape[0];
    *csz = t_shape[1];
    t_shape[0] = t_shape[1] = 0;
}
// the smallest of the caps on a launch's blocks: library-wide, the host thread's, and `share`
int persist_cap(int share) {
    int cap = PG_MAXB;
    for (int b : {g_persist_blocks, t_persist_blocks, share})
        if (b > 0 && b < cap) cap = b;
    return cap;
}
// CTAs of a one-cluster grid within the cap (0: a single block, no cluster)
int persist_one_cluster(int cap) { return cap >= 8 ? 8 : cap >= 4 ? 4 : cap >= 2 ? 2 : 0; }
int persist_thread_blocks(int n) {
    const int old = t_persist_blocks;
    if (n >= 0) t_persist_blocks = n;
    return old;
}

// The closing record of a launch: `rec` is the instance's landing place, which keeps the record of
// the solve before, so its error word is set before the copy and a copy or wait that failed, or a
// record that never landed, is no result.  1: arrived and sound, -1: not
static void record_arm(PGridHead *rec) { rec->err = PG_NO_RECORD; }
static int record_take(cudaError_t copy, cudaError_t wait, PGridHead *rec) {
    if (copy != cudaSuccess || wait != cudaSuccess) rec->err = PG_NO_RECORD;
    return rec->err ? -1 : 1;
}
// (into pinned memory: a copy to pageable memory waits for the solve inside the driver and
// holds up other threads' launches, eight diodes on eight threads 143 -> 159 ms)
int persist_record(const Ctx &c, const PGrid *g, PGridHead *out) {
    PGridHead *rec = c.pin ? c.pin : out;
    record_arm(rec);
    const cudaError_t copy = cudaMemcpyAsync(rec, g, sizeof(PGridHead), cudaMemcpyDeviceToHost, c.st);
    const cudaError_t wait = cudaStreamSynchronize(c.st);
    const int rc = record_take(copy, wait, rec);
    if (rec != out) *out = *rec;
    return rc;
}
int persist_record_probe(int copy, int wait, int arrives, unsigned err) {
    PGridHead rec{};                               // the solve before ended well
    rec.rec[0].status = 1;
    record_arm(&rec);
    if (arrives) rec.err = err;
    return record_take((cudaError_t)copy, (cudaError_t)wait, &rec);
}

// Launch the persistent solve `kind` of precision T on instance 0 of the context (n1: nodes of
// level 1).  Returns
// 1 when it ran (results in the Krylov records), 0 when the persistent path does not apply
// (the caller runs the per-pass path), -1 when a barrier wait ran out (the caller restores
// the start and runs the per-pass path; the persistent path is off from then on).
template <class T, int KIND>
static int persist_run(const Ctx &c, int n1, size_t smem, const PArgs &a, PGridHead *hres) {
    static KInfo info;                           // per instantiation, cached
    static std::mutex mu;
    KInfo ki;
    {
        std::lock_guard<std::mutex> lk(mu);
        KInfo &k = info;
        if (!k.fn || k.smem < smem) {
            k.fn = kfn<T, KIND>();
            k.smem = smem;
            k.blocks = occupancy(k.fn, smem);
            k.clusters[0] = cluster_occupancy(k.fn, smem, 8);
            k.clusters[1] = g_csz > 8 ? cluster_occupancy(k.fn, smem, 16) : 0;
        }
        ki = k;
    }
    int nb = ki.blocks;
    // small systems take a part of the GPU (about two nodes per thread), so that several
    // instances' solves can run side by side
    const int want = (c.maxN + 2 * PT_TPB - 1) / (2 * PT_TPB);
    if (want < nb) nb = want < 4 ? 4 : want;
    const int cap = persist_cap(c.pblocks);
    if (cap < nb) nb = cap;
    if (nb < 1) return 0;
    // Clusters.  A grid of at most 8 blocks becomes one cluster of 8 CTAs (under a cap below 8 of 4
    // or 2: a cap is a promise to the solves next to it), up to 31 blocks' worth one of 16: its barriers are cluster barriers, 0.3 us against 1.2-1.5 us for a grid barrier
    // (11,520 / 16,128 / 28,672 nodes FP64 38.9 / 39.9 / 45.3 -> 33.6 / 35.9 / 41.0 ms a sweep).  A larger grid is
    // a whole number of 16-CTA clusters, the first of which runs level 1 .. Ls-1 alone, while
    // level 1 has at most three (FP32: four) nodes a thread of that cluster: 64,000 nodes 82.5 ->
    // 78.0 ms, 180,000 96.6 -> 93.6 (FP32 89.1 -> 86.5), FP32 FinFET of 214,000 129.3 -> 127.0.
    // Beyond, the cluster's passes take longer than the whole grid's with its barriers, and level
    // 0 misses the SMs that no whole cluster covers (112 of 148 blocks): 230,400 nodes FP64 101.1
    // -> 103.1, 336,000 118.2 -> 124.9 (FP32 98.4 -> 103.2); clusters of 8 for that part lose
    // from 180,000 nodes on (101.2).  Only seven clusters of 16 fit the GPU: where fewer such
    // grids than plain ones run side by side, a batched resolve's workers take plain grids (six
    // of 36,864 nodes: 74 ms plain, 82 in clusters of 16), as do capped grids, which share the SMs by
    // blocks.  Nothing else of the process enters the choice: the order of the reductions follows
    // from the solve's size and the caller's own settings.
    PArgs aa = a;
    aa.csz = 0;
    aa.onecl = 0;
    aa.Lc = a.Ls;
    const bool capped = c.pblocks > 0 || t_persist_blocks > 0 || g_persist_blocks > 0;
    const int c16 = ki.clusters[1], per = sizeof(T) == 4 ? 4 : 3;
    int csz = 0, ncl = 1;
    if (g_clusters && ki.clusters[0] > 0 && nb <= 8) {
        csz = persist_one_cluster(cap);
    } else if (g_clusters == 2 && (c16 > 0 || ki.clusters[0] > 0)) {
        csz = c16 > 0 && cap >= 16 ? 16 : 8;
        ncl = std::max(1, std::min(nb / csz, csz > 8 ? c16 : ki.clusters[0]));
    } else if (g_clusters == 1 && c16 > 0 && !capped && n1 <= per * 16 * PT_TPB) {
        ncl = std::max(1, std::min(nb / 16, c16));
        if (2 * nb <= ki.blocks && ncl > 3) ncl = 3;        // two of these grids run side by side
        if (!c.batched || ki.blocks / nb <= c16 / ncl) csz = 16;
    }
    if (csz) {
        nb = ncl * csz;
        aa.csz = csz;
        aa.onecl = ncl == 1;
        if (ncl > 1) aa.Lc = g_clevel < a.Ls ? g_clevel : a.Ls;
    }
    PGrid *g = c.h.pgrid;
    cudaMemsetAsync(g, 0, 6 * sizeof(unsigned), c.st);      // counter, error word, work counters
    const DevP *dp = c.dP;
    if (g_trace && !g_trace_used) {              // the armed timeline records this launch only
        aa.trace = g_trace;
        aa.ntrace = g_trace_n;
        g_trace_used = 1;
    }
    void *args[] = {(void *)&dp, (void *)&aa};
    g_launches++;
    t_launches++;
    const int pid = sizeof(T) == 4 ? PF_PERSIST32 : PF_PERSIST;
    if (g_prof_on) prof_begin(pid, c.st);
    g_last_blocks = nb;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nb);
    cfg.blockDim = dim3(PT_TPB);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = g_coop;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = aa.csz; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = aa.csz ? 2 : 1;
    cudaError_t e = cudaLaunchKernelExC(&cfg, kfn<T, KIND>(), args);
    if (e != cudaSuccess && aa.csz) {            // no cluster launch here: plain cooperative grid
        cudaGetLastError();
        std::fprintf(stderr, "semisim-b200: cluster launch of the persistent solve refused (%s); without clusters "
                             "from now on\n", cudaGetErrorString(e));
        g_clusters = 0;
        aa.csz = 0;
        aa.onecl = 0;
        aa.Lc = aa.Ls;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelExC(&cfg, kfn<T, KIND>(), args);
    }
    if (g_prof_on) prof_end(pid, c.st, 0.0);
    if (e != cudaSuccess) {
        cudaGetLastError();
        std::fprintf(stderr, "semisim-b200: persistent solve launch failed (%s); per-pass solves from now on\n",
                     cudaGetErrorString(e));
        g_persist_broken = true;
        return 0;
    }
    persist_note(nb, aa.csz);
    const int rc = persist_record(c, g, hres);
    if (rc < 0) {
        std::fprintf(stderr, "semisim-b200: persistent solve abandoned (%s); per-pass solves from now on\n",
                     hres->err == 1 ? "a barrier wait ran out" : "its closing record did not arrive");
        g_persist_broken = true;
    }
    return rc;
}

// algorithmic bytes of one V-cycle of precision T (the passes the persistent kernel runs): a
// half sweep reads 6 couplings, pivot, right-hand side and the other colour and writes its
// own (10 words a node of its colour; the diagonal and own values too in a black update)
template <class T>
static double vcycle_bytes(const MGHost &mg, int Ls, int deep, int sweeps2) {
    double b = 0.0;
    for (int L = 0; L < Ls; L++) {
        const double half = 0.5 * mg.maxN[L] * sizeof(T);
        const double twice = (L < deep && sweeps2) ? 2.0 * (10.0 + 12.0) : 0.0;
        b += half * (10.0 + 10.0 + 10.25 + 11.25 + 13.25 + 10.0 + twice);
    }
    b += 2.0 * mg.maxN[Ls] * sizeof(T);             // b in, x out of the shared-memory levels
    return b;
}

// algorithmic bytes of the in-kernel hierarchy set-up of precision T
template <class T>
static double setup_bytes(const MGHost &mg) {
    const double w = sizeof(T) / 8.0;
    double b = sizeof(T) == 4 ? mg.maxN[0] * kProfBytesPerNode[PF_CONVERT32] : 0.0;
    for (int L = 0; L < mg.maxlev - 1; L++)
        b += mg.maxN[L] * w * (kProfBytesPerNode[PF_WEIGHTS] + kProfBytesPerNode[PF_GALERKIN] +
                               kProfBytesPerNode[PF_ILU_DIAG]);
    return b;
}

// small-level plan of precision T for the persistent kernels: the first level at or below
// the small-level size whose data fits the opt-in shared memory (never level 0)
template <class T>
static int persist_plan(const Ctx &c, const MGHost &mg, size_t *smem) {
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const size_t cap = optin > 16384 ? (size_t)optin - 16384 : 0;
    *smem = 0;
    if (mg.maxlev < 2) return -1;
    vcycle_knobs_init();
    const int lim = c.small_nodes > 0 ? c.small_nodes : g_small_nodes;
    int L = 1;
    while (L < mg.maxlev - 1 && mg.maxN[L] > lim) L++;
    auto bytes = [&](int Ls) {
        size_t b = 0;
        for (int q = Ls; q < mg.maxlev; q++) {
            const int hx = (((mg.maxNx[q] + 1) / 2) + 1) & ~1, H = hx * mg.maxRows[q], ap = (2 * H + 31) & ~31;
            b += ssm_level<T>(H, ap, mg.maxN[q], q == mg.maxlev - 1);
        }
        return b;
    };
    while (L < mg.maxlev - 1 && bytes(L) > cap) L++;
    if (bytes(L) > cap || mg.maxlev - L > 15) return -1;    // (one hardware barrier per level)
    *smem = bytes(L);
    return L;
}

// Persistent forms of the solves of kernels_la.cu; k: the starting Krylov record (it travels
// with the launch's parameters) and the closing one (it comes back with the launch's status:
// one copy and one wait a solve).  Each returns 1 (done), 0 (not applicable: nothing was changed) or -1 (abandoned: the
// caller restores the start and uses the per-pass solve).
int persist_pcg(const Ctx &c, const MGHost &mg, int mixed, KrylovS &k) {
    if (c.ninst != 1 || !c.h.pwd || !persist_enabled()) return 0;
    size_t smem = 0;
    PArgs a{};
    a.Ls = mixed ? persist_plan<float>(c, mg, &smem) : persist_plan<double>(c, mg, &smem);
    if (a.Ls < 1) return 0;
    a.qsign = 0;
    a.deep = g_deep_levels;
    a.sweeps2 = 0;                              // one application (MG_OVER, solver_ctx.h)
    a.alpha = mg.alpha_p;
    a.barmode = g_barmode;
    a.rec[0] = k;
    PGridHead h{};
    const int rc = mixed ? persist_run<float, PK_PCG>(c, mg.maxN[1], smem, a, &h)
                         : persist_run<double, PK_PCG>(c, mg.maxN[1], smem, a, &h);
    if (rc == 1) k = h.rec[0];
    if (rc == 1 && g_prof_on) {
        const double vb = mixed ? vcycle_bytes<float>(mg, a.Ls, a.deep, a.sweeps2)
                                : vcycle_bytes<double>(mg, a.Ls, a.deep, a.sweeps2);
        const double kb = (mixed ? 0.5 : 1.0) * (kProfBytesPerNode[PF_KRY_SPMV_DOT] + 2 * kProfBytesPerNode[PF_KRY_UPDATE] +
                                                 kProfBytesPerNode[PF_KRY_DOT]);
        const double sb = mixed ? setup_bytes<float>(mg) : setup_bytes<double>(mg);
        prof_set_last(mixed ? PF_PERSIST32 : PF_PERSIST, sb + h.vcycles * vb + h.iters * kb * c.maxN);
    }
    return rc;
}
int persist_bicg(const Ctx &c, const MGHost &mg, KrylovS &k, int qsign) {
    if (c.ninst != 1 || !c.h.pwd || !persist_enabled()) return 0;
    size_t smem = 0;
    PArgs a{};
    a.Ls = persist_plan<double>(c, mg, &smem);
    if (a.Ls < 1) return 0;
    a.qsign = qsign;
    a.deep = g_deep_levels;
    a.sweeps2 = g_l0_sweeps > 1;
    a.alpha = mg.alpha;
    a.barmode = g_barmode;
    a.rtol = k.rtol;
    a.atol = k.atol;
    a.rec[0] = k;
    PGridHead h{};
    const int rc = persist_run<double, PK_BICG>(c, mg.maxN[1], smem, a, &h);
    if (rc == 1) k = h.rec[0];
    if (rc == 1 && g_prof_on) {
        const double vb = vcycle_bytes<double>(mg, a.Ls, a.deep, a.sweeps2);
        const double kb = 2 * kProfBytesPerNode[PF_KRY_SPMV_DOT] + 4 * kProfBytesPerNode[PF_KRY_UPDATE];
        prof_set_last(PF_PERSIST, setup_bytes<double>(mg) + h.vcycles * vb +
                                      (h.iters * kb + kProfBytesPerNode[PF_KRY_INIT]) * c.maxN);
    }
    return rc;
}
int persist_refined(const Ctx &c, const MGHost &mg, int maxsteps, int *steps, int qsign, const KrylovS &inner, KrylovS &k) {
    if (c.ninst != 1 || !c.h.pwd || !persist_enabled()) return 0;
    size_t smem = 0;
    PArgs a{};
    a.Ls = persist_plan<float>(c, mg, &smem);
    if (a.Ls < 1) return 0;
    a.qsign = qsign;
    a.deep = g_deep_levels;
    a.sweeps2 = g_l0_sweeps > 1;
    a.alpha = mg.alpha;
    a.barmode = g_barmode;
    a.maxsteps = maxsteps;
    a.rec[0] = inner;
    a.rec[1] = k;
    PGridHead h{};
    const int rc = persist_run<float, PK_REFINED>(c, mg.maxN[1], smem, a, &h);
    if (rc == 1) {
        k = h.rec[1];
        *steps = h.steps;
        if (g_prof_on) {
            const double vb = vcycle_bytes<float>(mg, a.Ls, a.deep, a.sweeps2);
            const double kb = 0.5 * (2 * kProfBytesPerNode[PF_KRY_SPMV_DOT] + 4 * kProfBytesPerNode[PF_KRY_UPDATE]);
            prof_set_last(PF_PERSIST32, setup_bytes<float>(mg) + h.vcycles * vb +
                                            (h.iters * kb + (h.steps + 1) * kProfBytesPerNode[PF_REFINE]) * c.maxN);
        }
    }
    return rc;
}

// Barrier timeline of the next persistent launch (test and measurement hook): n > 0 arms a
// timeline of n barriers; n == 0 copies the recorded one to out (3 n values: first arrival,
// last arrival, release seen by block 0, globaltimer ns; unused barriers keep ~0, 0, 0),
// disarms it and returns the blocks of that launch.
int persist_trace(int n, unsigned long long *out, int *blocks) {
    static int nmax = 0;
    if (n > 0) {
        if (g_trace) cudaFree(g_trace);
        g_trace = nullptr;
        if (cudaMalloc(&g_trace, sizeof(unsigned long long) * 3 * n) != cudaSuccess) { cudaGetLastError(); return -1; }
        std::vector<unsigned long long> init(3 * (size_t)n, 0ull);
        for (int q = 0; q < n; q++) init[3 * q] = ~0ull;
        cudaMemcpy(g_trace, init.data(), init.size() * sizeof(unsigned long long), cudaMemcpyHostToDevice);
        g_trace_n = nmax = n;
        g_trace_used = 0;
        return 0;
    }
    if (!g_trace) return -1;
    cudaDeviceSynchronize();
    if (out) cudaMemcpy(out, g_trace, sizeof(unsigned long long) * 3 * nmax, cudaMemcpyDeviceToHost);
    cudaFree(g_trace);
    g_trace = nullptr;
    g_trace_n = 0;
    if (blocks) *blocks = g_last_blocks;
    return g_trace_used;
}

// Run the bounded-wait test on the instance's barrier record with `nb` blocks (>= 2):
// returns the error word (1 expected) and the blocks that reported ok = 0 in *gave_up
// (nb - 1 expected), or -1 when the launch failed.
int persist_timeout_probe(const Ctx &c, int nb, double wait_s, int *gave_up) {
    if (nb < 2 || nb > 64) return -1;
    int *ok = nullptr;
    if (cudaMalloc(&ok, nb * sizeof(int)) != cudaSuccess) { cudaGetLastError(); return -1; }
    cudaMemsetAsync(ok, 0xff, nb * sizeof(int), c.st);
    PGrid *g = c.h.pgrid;
    cudaMemsetAsync(g, 0, 6 * sizeof(unsigned), c.st);
    unsigned long long wn = (unsigned long long)(wait_s * 1e9);
    void *args[] = {(void *)&g, (void *)&wn, (void *)&ok};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void *)k_pg_timeout_probe, dim3(nb), dim3(32), args, 0, c.st);
    int rc = -1;
    if (e == cudaSuccess) {
        unsigned err = 0;
        std::vector<int> h(nb);
        cudaMemcpyAsync(&err, &g->err, sizeof(unsigned), cudaMemcpyDeviceToHost, c.st);
        cudaMemcpyAsync(h.data(), ok, nb * sizeof(int), cudaMemcpyDeviceToHost, c.st);
        if (cudaStreamSynchronize(c.st) == cudaSuccess) {
            int n0 = 0;
            for (int q = 0; q < nb - 1; q++) n0 += h[q] == 0;
            *gave_up = n0;
            rc = (int)err;
        }
    } else {
        cudaGetLastError();
    }
    cudaFree(ok);
    return rc;
}

}  // namespace ss
