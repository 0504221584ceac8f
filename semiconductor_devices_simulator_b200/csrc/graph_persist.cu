// Persistent linear solves of general (graph) meshes: one cooperative launch runs a whole
// PCG or BiCGSTAB solve preconditioned by the aggregation multigrid - the hierarchy's
// set-up, every iteration and V-cycle with the multicolour D-ILU(0) smoother, the dense
// coarsest inverse and its solves - with barriers between the dependent passes instead of one
// kernel launch per colour and a host round trip per dot product (pcg_graph / bicg_graph in
// graph.cu, which this replaces when it applies).
//
// What bounds it: the graphs in use have 1,000 - 100,000 nodes, so a pass moves little and a
// solve costs (passes) x (barrier + latency of one pass's dependent loads).  Therefore:
//   * the solve keeps its own copy of every level with the nodes ordered by colour and each
//     row's slots split into the couplings to earlier colours (first DL) and to later ones
//     (last DU), padded with zero couplings to the node itself: a colour's sweep reads
//     contiguous rows and needs neither colours nor tests (slot by slot in mesh order with a
//     colour look-up per neighbour a V-cycle on 7,200 nodes took 288 us, now 120 us);
//   * set-up in the same launch: Galerkin sums gathered per coarse coupling, the D-ILU pivots of
//     all levels side by side (colour c of level L in stage L + c), the dense inverse spread over
//     up to 8 blocks in registers, four columns per barrier (the separate launches took 0.85 ms
//     a solve, 0.49 ms of it one block's inverse, now 0.14 ms);
//   * meshes that fit one cluster of 8 blocks use its hardware barrier (0.3 us against 1.3 us
//     for a grid barrier);
//   * levels of at most GP_SMALL nodes below the mesh: block 0 alone with block barriers (the
//     other blocks wait at the next barrier);
//   * fused passes: the residual summed straight into the aggregates on the way down; on the
//     way up the forward sweep takes the residual as it goes, and the backward sweep adds the
//     correction; one reduction per PCG iteration, x, r and the next p of BiCGSTAB in one pass
//     (as in kernels_persist.cu).
// The Krylov scalars are reduced in every block (persist_common.cuh), so the stop decisions
// are the same in every block; the stop rules are the reference's (gpcg / gbicgstab,
// semiconductor_3d.c:2682-2714 with bicgstab_core's rules :2244-2320).
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "persist_common.cuh"
#include "prof.h"
#include "solver_ctx.h"

namespace ss {

constexpr int GP_TPB = 512;
constexpr int GP_MAXC = 64;         // most colours of a level
constexpr int GP_SMALL = 4096;      // levels at or below this size run in block 0
constexpr int GP_MAXL = 16;         // most levels (the level table lives in shared memory)
constexpr int GP_CL = 8;            // blocks of a one-cluster launch, and of the dense inverse
constexpr int GP_CLUSTER_N = 16384; // meshes up to this size run as one cluster (2 nodes a thread and colour pass
                                    //   at 2 colours; above it more blocks pay for the dearer barrier)
constexpr int GP_INV_REG = 160;     // the dense inverse in registers up to this size (10 columns a lane)

// one level as the persistent kernel sees it: position t of the colour order, slot q of row
// t at q*N + t
struct PGLev {
    int N, S, DL, ncolor;
    const int *col;                   // neighbour's position (padding: t itself)
    const int *src;                   // level 0: the mesh's ELL entry of the slot (-1: padding)
    const int *rev;                   // of the first DL slots: the reverse coupling's entry
    double *val, *diag, *dil, *pw, *ph, *x, *b;
    const int *node;                  // level 0: mesh node of the position
    double *w;                        // level 0: row weights
    const int *agg, *mrp, *mem;       // towards the next level, all in positions
    // gather lists of the next level's operator: entries of this level that sum into slot q of
    // coarse row I (eptr[I * Sc + q] ..) and, inside the aggregate, into its diagonal (dptr[I] ..)
    const int *eptr, *elist, *dptr, *dlist;
    double *inv;                      // coarsest level: dense inverse
    int cptr[GP_MAXC + 1];
};
struct GPArgs {
    const PGLev *lev;
    double *prow;        // 2 x 4 pivot rows of the dense inverse
    int nl, Ls;          // levels; the first one block 0 runs alone
    int kind;            // 0 PCG, 1 BiCGSTAB
    int ilu_only;        // BiCGSTAB preconditioned by the mesh level's D-ILU(0) alone
    int qsign;           // Slotboom weights: 0 none, +1 electrons, -1 holes
    int onecl;
    double alpha, rtol, atol;
    KrylovS rec;         // starting record
};

// the threads that run a level: the whole grid, or block 0 alone
struct GE {
    int tid, nth;
    bool blk;
};
__device__ __forceinline__ bool ge_sync(PS &s, const GE &e) {
    if (e.blk) { __syncthreads(); return true; }
    return pg_sync(s);
}
#define GP_SYNC(E)                     \
    do {                               \
        if (!ge_sync(s, (E))) return false; \
    } while (0)

// Lanes per row (log2): as many of 8, 4 or 2 as still leave the pass one trip over the rows - its
// loads then cost one round trip for the columns and one for the values instead of one per batch
// of slots - and one thread a row where the rows fill the threads anyway.
__device__ __forceinline__ int gp_lanes(int rows, int nth) {
    return 8 * rows <= nth ? 3 : (4 * rows <= nth ? 2 : (2 * rows <= nth ? 1 : 0));
}
__device__ __forceinline__ double gp_fold(double v, int gsh) {
    if (gsh > 2) v += __shfl_xor_sync(0xffffffffu, v, 4);
    if (gsh > 1) v += __shfl_xor_sync(0xffffffffu, v, 2);
    if (gsh) v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}
// this lane's part of the sum over the slots q0 .. q1-1 of row t of a_tj x_j, NB
// slots' loads in flight; LO: with z, also the part of the first DL slots
template <bool LO, int NB>
__device__ __forceinline__ double gp_part(const PGLev &v, int q0, int q1, int t, const double *x, const double *z,
                                          int lane, int gsh, double &lo) {
    double sum = 0.0;
    lo = 0.0;
    const int g = 1 << gsh;
    for (int q = q0 + lane; q < q1; q += NB * g) {
        int j[NB];
        double a[NB];
#pragma unroll
        for (int i = 0; i < NB; i++) {
            const int w = q + i * g;
            const size_t e = (size_t)(w < q1 ? w : q) * v.N + t;
            j[i] = v.col[e];
            a[i] = w < q1 ? v.val[e] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < NB; i++) {
            sum += a[i] * x[j[i]];
            if (LO) lo += (q + i * g < v.DL ? a[i] : 0.0) * z[j[i]];
        }
    }
    return sum;
}

// D-ILU(0) solve z = M^-1 r of one level (gilu_apply, semiconductor_3d.c:2563-2593): forward
// colours then backward colours.  UP: r is the residual b - A x, taken as the forward sweep
// goes, and the backward sweep ends with x += z.
template <bool UP>
__device__ bool gp_ilu(PS &s, const GE &e, const PGLev &Hr, const double *b, double *z, double *x) {
    const PGLev &H = Hr;
    const int nc = H.ncolor;
    for (int c = 0; c < nc; c++) {
        const int c0 = H.cptr[c], rows = H.cptr[c + 1] - c0, gsh = gp_lanes(rows, e.nth);
        const int lane = e.tid & ((1 << gsh) - 1), n = ((rows << gsh) + 31) & ~31;
        for (int u = e.tid; u < n; u += e.nth) {
            const int t = c0 + (u >> gsh);
            const bool ok = (u >> gsh) < rows;
            double sum = 0.0, lo = 0.0, bt = 0.0, dil = 0.0, xt = 0.0;
            if (ok) {
                bt = b[t];
                dil = H.dil[t];
                if (UP) {
                    xt = x[t];
                    sum = gp_part<true, 4>(H, 0, H.S, t, x, z, lane, gsh, lo) + lo;
                    if (lane == 0) sum += H.diag[t] * xt;
                } else if (c) {
                    sum = gp_part<false, 4>(H, 0, H.DL, t, z, nullptr, lane, gsh, lo);
                }
            }
            sum = gp_fold(sum, gsh);
            if (ok && lane == 0) {
                const double y = (bt - sum) * dil;
                z[t] = y;
                if (UP && c == nc - 1) x[t] = xt + y;      // (the last colour has no later ones)
            }
        }
        GP_SYNC(e);
    }
    for (int c = nc - 2; c >= 0; c--) {
        const int c0 = H.cptr[c], rows = H.cptr[c + 1] - c0, gsh = gp_lanes(rows, e.nth);
        const int lane = e.tid & ((1 << gsh) - 1), n = ((rows << gsh) + 31) & ~31;
        for (int u = e.tid; u < n; u += e.nth) {
            const int t = c0 + (u >> gsh);
            const bool ok = (u >> gsh) < rows;
            double sum = 0.0, lo, zt = 0.0, dil = 0.0, xt = 0.0;
            if (ok) {
                zt = z[t];
                dil = H.dil[t];
                if (UP) xt = x[t];
                sum = gp_part<false, 4>(H, H.DL, H.S, t, z, nullptr, lane, gsh, lo);
            }
            sum = gp_fold(sum, gsh);
            if (ok && lane == 0) {
                const double y = zt - sum * dil;
                z[t] = y;
                if (UP) x[t] = xt + y;
            }
        }
        GP_SYNC(e);
    }
    return true;
}

// row t of A x in every lane of the row's group
__device__ __forceinline__ double gp_apply(const PGLev &H, const double *x, int t, bool ok, int lane, int gsh) {
    double sum = 0.0, lo;
    if (ok) {
        sum = gsh ? gp_part<false, 4>(H, 0, H.S, t, x, nullptr, lane, gsh, lo)
                  : gp_part<false, 8>(H, 0, H.S, t, x, nullptr, lane, gsh, lo);
        if (lane == 0) sum += H.diag[t] * x[t];
    }
    return gp_fold(sum, gsh);
}
// y = A x on the mesh level; f(t, y_t) once per row
template <class F>
__device__ __forceinline__ void gp_spmv(const PGLev &H, const PS &s, const double *x, F f) {
    const int gsh = gp_lanes(H.N, s.nth), lane = s.tid & ((1 << gsh) - 1), n = ((H.N << gsh) + 31) & ~31;
    for (int u = s.tid; u < n; u += s.nth) {
        const int t = u >> gsh;
        const bool ok = t < H.N;
        const double y = gp_apply(H, x, t, ok, lane, gsh);
        if (ok && lane == 0) f(t, y);
    }
}

// the way down at level L: pre-smoothing x = M^-1 b from x = 0, the weighted residual in z,
// and its sums over the aggregates of level L + 1 (8 lanes each)
__device__ bool gp_down(PS &s, const GE &e, const PGLev &H, const PGLev &Hc, const double *b, double *x, double *z,
                        const double *w) {
    if (!gp_ilu<false>(s, e, H, b, x, nullptr)) return false;
    {
        const int gsh = gp_lanes(H.N, e.nth), lane = e.tid & ((1 << gsh) - 1), n = ((H.N << gsh) + 31) & ~31;
        for (int u = e.tid; u < n; u += e.nth) {
            const int t = u >> gsh;
            const bool ok = t < H.N;
            const double y = gp_apply(H, x, t, ok, lane, gsh);
            if (ok && lane == 0) z[t] = w ? w[t] * (b[t] - y) : b[t] - y;
        }
    }
    GP_SYNC(e);
    const int lane = e.tid & 7, n8 = (Hc.N * 8 + 31) & ~31;
    for (int u = e.tid; u < n8; u += e.nth) {
        const int I = u >> 3;
        double sum = 0.0;
        if (I < Hc.N)
            for (int q = H.mrp[I] + lane; q < H.mrp[I + 1]; q += 8) sum += z[H.mem[q]];
        sum = gp_fold(sum, 3);
        if (lane == 0 && I < Hc.N) Hc.b[I] = sum;
    }
    GP_SYNC(e);
    return true;
}

// the way up at level L: x += alpha pw xc, then one D-ILU(0) correction from its residual
__device__ bool gp_up(PS &s, const GE &e, const PGLev &H, const PGLev &Hc, const double *b, double *x, double *z,
                      double al) {
    const double *xc = Hc.x;
    for (int t = e.tid; t < H.N; t += e.nth) x[t] += al * H.pw[t] * xc[H.agg[t]];
    GP_SYNC(e);
    return gp_ilu<true>(s, e, H, b, z, x);
}

// x = inverse b on the coarsest level (one warp per row)
__device__ bool gp_coarse(PS &s, const GE &e, const PGLev &v) {
    const int lane = threadIdx.x & 31, n = v.N;
    for (int r = e.tid >> 5; r < n; r += e.nth >> 5) {
        double sum = 0.0;
        for (int q = lane; q < n; q += 32) sum += v.inv[(size_t)r * n + q] * v.b[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
        if (lane == 0) v.x[r] = sum;
    }
    GP_SYNC(e);
    return true;
}

// one V-cycle z = M^-1 r on the mesh level (gvcycle, semiconductor_3d.c:2654-2680); zw: a
// work vector of the mesh level
__device__ __noinline__ bool gp_vcycle(PS &s, const GPArgs &a, const double *b0, double *x0, double *zw) {
    const GE grid{s.tid, s.nth, false};
    if (a.ilu_only) return gp_ilu<false>(s, grid, a.lev[0], b0, x0, nullptr);
    const int nl = a.nl, Ls = a.Ls;
    auto B = [&](int L) { return L ? a.lev[L].b : b0; };
    auto X = [&](int L) { return L ? a.lev[L].x : x0; };
    // (levels below the mesh keep their residuals and the post-smoothing's z in ph, which is free
    // after the set-up)
    auto Z = [&](int L) { return L ? a.lev[L].ph : zw; };
    const int Lg = Ls < nl - 1 ? Ls : nl - 1;            // levels 0 .. Lg-1: the whole grid
    for (int L = 0; L < Lg; L++)
        if (!gp_down(s, grid, a.lev[L], a.lev[L + 1], B(L), X(L), Z(L), L ? nullptr : (a.qsign ? a.lev[0].w : nullptr)))
            return false;
    if (Ls <= nl - 1) {
        if (blockIdx.x == 0) {                           // the small levels: block 0 alone
            const GE blk{(int)threadIdx.x, (int)blockDim.x, true};
            for (int L = Ls; L < nl - 1; L++) gp_down(s, blk, a.lev[L], a.lev[L + 1], B(L), X(L), Z(L), nullptr);
            gp_coarse(s, blk, a.lev[nl - 1]);
            for (int L = nl - 2; L >= Ls; L--) gp_up(s, blk, a.lev[L], a.lev[L + 1], B(L), X(L), Z(L), a.alpha);
        }
        if (!pg_sync(s)) return false;
    } else if (!gp_coarse(s, grid, a.lev[nl - 1])) {
        return false;
    }
    for (int L = Lg - 1; L >= 0; L--)
        if (!gp_up(s, grid, a.lev[L], a.lev[L + 1], B(L), X(L), Z(L), a.alpha)) return false;
    if (blockIdx.x == 0 && threadIdx.x == 0) s.g->vcycles++;
    return true;
}

// ---------------------------------------------------------------- set-up
// Slotboom weights towards the next level: pw = exp(ph - max over the aggregate) (g_weights,
// semiconductor_3d.c:2621-2642)
__device__ __forceinline__ double gp_ph(const DevP &P, const PGLev &f, int L, int t, int qsign) {
    if (L) return f.ph[t];
    const int k = f.node[t];
    const uint32_t fl = P.flags[k];
    if (fl_kind(fl) != K_SEMI || fl_fix(fl)) return PH_NONE;
    return qsign > 0 ? P.phin[k] / P.VTref : -P.phip[k] / P.VTref;
}
__device__ void gp_weights(const DevP &P, const PGLev &f, const PGLev &c, int L, int qsign, int tid, int nth) {
    if (!qsign) {
        for (int t = tid; t < f.N; t += nth) f.pw[t] = 1.0;
        return;
    }
    const int lane = tid & 7, n8 = (c.N * 8 + 31) & ~31;      // 8 lanes per aggregate
    for (int u = tid; u < n8; u += nth) {
        const int I = u >> 3, q0 = I < c.N ? f.mrp[I] : 0, q1 = I < c.N ? f.mrp[I + 1] : 0;
        double mx = PH_NONE;
        for (int q = q0 + lane; q < q1; q += 8) mx = fmax(mx, gp_ph(P, f, L, f.mem[q], qsign));
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0 && I < c.N) c.ph[I] = mx;
        for (int q = q0 + lane; q < q1; q += 8) {
            const int t = f.mem[q];
            const double p = gp_ph(P, f, L, t, qsign), e = (p <= 0.5 * PH_NONE) ? -800.0 : p - mx;
            f.pw[t] = e < -700.0 ? 0.0 : exp(e);
        }
    }
}
// coarse operator P^T W A P (g_galerkin, semiconductor_3d.c:2575-2594), 8 lanes per coarse
// row: a lane sums whole couplings from their gather lists; a row of identity rows only stays
// an identity row
__device__ __forceinline__ double gp_gather(const PGLev &f, const int *list, int p0, int p1, int st, const double *w) {
    double sum = 0.0;
    for (int p = p0; p < p1; p += 4 * st) {
        int e[4], j[4];
        double a[4], c[4];
#pragma unroll
        for (int i = 0; i < 4; i++) e[i] = list[p + i * st < p1 ? p + i * st : p];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            j[i] = f.col[e[i]];
            a[i] = p + i * st < p1 ? f.val[e[i]] : 0.0;
            c[i] = w ? w[e[i] % f.N] : 1.0;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) sum += c[i] * a[i] * f.pw[j[i]];
    }
    return sum;
}
__device__ void gp_galerkin(const PGLev &f, const PGLev &c, const double *w, int tid, int nth) {
    const int lane = tid & 7, n8 = (c.N * 8 + 31) & ~31;
    for (int u = tid; u < n8; u += nth) {
        const int I = u >> 3;
        bool any = false;
        double dg = 0.0;
        if (I < c.N) {
            for (int q = lane; q < c.S; q += 8) {
                const double sum = gp_gather(f, f.elist, f.eptr[I * c.S + q], f.eptr[I * c.S + q + 1], 1, w);
                c.val[(size_t)q * c.N + I] = sum;
                any = any || sum != 0.0;
            }
            dg = gp_gather(f, f.dlist, f.dptr[I] + lane, f.dptr[I + 1], 8, w);
            for (int q = f.mrp[I] + lane; q < f.mrp[I + 1]; q += 8) {
                const int t = f.mem[q];
                dg += (w ? w[t] : 1.0) * f.diag[t] * f.pw[t];
            }
        }
        dg = gp_fold(dg, 3);
        const unsigned m = __ballot_sync(0xffffffffu, any);
        if (lane == 0 && I < c.N) {
            const bool none = ((m >> (threadIdx.x & 24)) & 255u) == 0u;
            c.diag[I] = dg == 0.0 && none ? 1.0 : dg;
        }
    }
}
// D-ILU(0) pivots of one colour: D_i = a_ii - sum over earlier colours a_ij a_ji / D_j, guarded
// as the reference guards its pivots (gilu_factor, semiconductor_3d.c:2533-2551); reciprocals
__device__ void gp_pivots(const PGLev &v, int c, int tid, int nth) {
    const int c0 = v.cptr[c], rows = v.cptr[c + 1] - c0, gsh = gp_lanes(rows, nth), g = 1 << gsh;
    const int lane = tid & (g - 1), n = ((rows << gsh) + 31) & ~31;
    for (int u = tid; u < n; u += nth) {
        const int t = c0 + (u >> gsh);
        const bool ok = (u >> gsh) < rows;
        double sum = 0.0;
        if (ok && c)
#pragma unroll 2
            for (int q = lane; q < v.DL; q += g) {
                const size_t e = (size_t)q * v.N + t;
                const int j = v.col[e];
                const double x = v.val[e] * v.val[v.rev[e]] * v.dil[j];
                sum += j != t ? x : 0.0;
            }
        sum = gp_fold(sum, gsh);
        if (ok && lane == 0) {
            const double a = v.diag[t];
            double d = a - sum;
            if (!(d > 1e-8 * fabs(a))) d = a;
            if (!(d != 0.0)) d = 1.0;
            v.dil[t] = 1.0 / d;
        }
    }
}
// Dense inverse of the coarsest level by Gauss-Jordan on the diagonal pivots (tiny ones set to
// 1e-300 as semiconductor_3d.c:2620 does).  No row interchanges: what leaves a node enters its
// neighbours, so with the row scaling taken out the columns of these systems sum to what
// recombination, exchange and contacts take (>= 0), their couplings are not positive, and both
// survive the sums over aggregates, the prolongation's weights (>= 0) and elimination.  The largest
// entry of a pivot column is thus its diagonal, which partial pivoting would take too (checked on
// diode, MOSFET and tunnelling systems by test_gpu_graph_coarse_dominance.py).
// Up to GP_INV_REG unknowns: nbk blocks own rb rows each, 16 lanes hold a row in registers.
// Four columns C at a time: their owner publishes the four rows P as they are, and after one
// barrier every row takes  row -= g P  with g = row_C D^-1, D the 4x4 pivot block (columns C
// become -g); the pivot rows become D^-1 P.
__device__ __forceinline__ void inv4(const double (&m)[16], double (&o)[16]) {
    // through 2x2 blocks [A B; C E]: S = E - C A^-1 B
    auto inv2 = [](const double *a, double *r) {
        double d = a[0] * a[3] - a[1] * a[2];
        d = 1.0 / (fabs(d) > 1e-300 ? d : 1e-300);
        r[0] = a[3] * d; r[1] = -a[1] * d; r[2] = -a[2] * d; r[3] = a[0] * d;
    };
    auto mul2 = [](const double *a, const double *b, double *r) {
        r[0] = a[0] * b[0] + a[1] * b[2]; r[1] = a[0] * b[1] + a[1] * b[3];
        r[2] = a[2] * b[0] + a[3] * b[2]; r[3] = a[2] * b[1] + a[3] * b[3];
    };
    const double A[4] = {m[0], m[1], m[4], m[5]}, B[4] = {m[2], m[3], m[6], m[7]}, C[4] = {m[8], m[9], m[12], m[13]},
                 E[4] = {m[10], m[11], m[14], m[15]};
    double Ai[4], CA[4], AB[4], S[4], Si[4], t[4], u[4];
    inv2(A, Ai);
    mul2(C, Ai, CA);
    mul2(Ai, B, AB);
    mul2(CA, B, t);
#pragma unroll
    for (int q = 0; q < 4; q++) S[q] = E[q] - t[q];
    inv2(S, Si);
    mul2(AB, Si, t);                              // A^-1 B S^-1
    mul2(Si, CA, u);                              // S^-1 C A^-1
    double w[4];
    mul2(t, CA, w);
    o[0] = Ai[0] + w[0]; o[1] = Ai[1] + w[1]; o[4] = Ai[2] + w[2]; o[5] = Ai[3] + w[3];
    o[2] = -t[0]; o[3] = -t[1]; o[6] = -t[2]; o[7] = -t[3];
    o[8] = -u[0]; o[9] = -u[1]; o[12] = -u[2]; o[13] = -u[3];
    o[10] = Si[0]; o[11] = Si[1]; o[14] = Si[2]; o[15] = Si[3];
}
__device__ __noinline__ bool gp_invert(PS &s, const GPArgs &a, const PGLev &v) {
    constexpr int NI = GP_INV_REG / 16;
    const int n = v.N, nb = gridDim.x, nbk = nb < GP_CL ? nb : GP_CL;
    const int rb = (((n + nbk - 1) / nbk) + 3) & ~3;
    const int lane = threadIdx.x & 15, lr = threadIdx.x >> 4, r = blockIdx.x * rb + lr;
    if (n <= GP_INV_REG && rb <= GP_TPB / 16) {
        const bool own = (int)blockIdx.x < nbk && lr < rb && r < n;
        double x[NI];
#pragma unroll
        for (int i = 0; i < NI; i++) x[i] = 0.0;
        if (own) {
            for (int q = 0; q < v.S; q++) {
                const size_t e = (size_t)q * n + r;
                const int j = v.col[e];
                const double y = j != r ? v.val[e] : 0.0;
#pragma unroll
                for (int i = 0; i < NI; i++)
                    if (j == lane + 16 * i) x[i] += y;
            }
#pragma unroll
            for (int i = 0; i < NI; i++)
                if (r == lane + 16 * i) x[i] += v.diag[r];
        }
        __shared__ double sp[4 * GP_INV_REG];
        int buf = 0;
        for (int c0 = 0; c0 < n; c0 += 4) {
            const int cn = min(4, n - c0);
            double *pr = a.prow + (size_t)buf * 4 * GP_INV_REG;
            buf ^= 1;
            if (own && r >= c0 && r < c0 + cn)
#pragma unroll
                for (int i = 0; i < NI; i++) pr[(r - c0) * GP_INV_REG + lane + 16 * i] = x[i];
            if (!pg_sync(s)) return false;
            if ((int)blockIdx.x < nbk)
                for (int q = threadIdx.x; q < 4 * GP_INV_REG; q += GP_TPB) sp[q] = __ldcg(pr + q);
            __syncthreads();                                       // (the next barrier ends the reads of sp)
            if ((threadIdx.x >> 5) * 2 >= rb) continue;            // a warp without rows
            double m[16], di[16], f[4], g[4];
            if (cn == 4) {
#pragma unroll
                for (int p = 0; p < 4; p++)
#pragma unroll
                    for (int q = 0; q < 4; q++) m[4 * p + q] = sp[p * GP_INV_REG + c0 + q];
            } else {
#pragma unroll
                for (int p = 0; p < 4; p++)
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        m[4 * p + q] = p < cn && q < cn ? sp[p * GP_INV_REG + c0 + q] : (p == q ? 1.0 : 0.0);
            }
            inv4(m, di);
            // row_C: the columns C lie in four lanes (c0 & 15) .. + 3 of one register
            double xc = 0.0;
#pragma unroll
            for (int i = 0; i < NI; i++) xc = i == (c0 >> 4) ? x[i] : xc;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                f[q] = __shfl_sync(0xffffffffu, xc, (c0 & 15) + q, 16);
                if (q >= cn) f[q] = 0.0;
            }
            const int pv = own && r >= c0 && r < c0 + cn ? r - c0 : -1;
            if (pv >= 0)                                           // a pivot row: 0 - (-D^-1) P
#pragma unroll
                for (int q = 0; q < 4; q++) f[q] = q == pv ? -1.0 : 0.0;
#pragma unroll
            for (int q = 0; q < 4; q++)
                g[q] = f[0] * di[q] + f[1] * di[4 + q] + f[2] * di[8 + q] + f[3] * di[12 + q];
            const int qc = lane - (c0 & 15);                       // this lane's column of C, if 0 .. 3
            const double gc = qc == 0 ? g[0] : (qc == 1 ? g[1] : (qc == 2 ? g[2] : g[3]));
#pragma unroll
            for (int i = 0; i < NI; i++) {
                if (16 * i >= n) break;
                const double *p = sp + lane + 16 * i;              // (rows past cn have g = 0)
                double y = pv >= 0 ? 0.0 : x[i];
                y -= g[0] * p[0];
                y -= g[1] * p[GP_INV_REG];
                y -= g[2] * p[2 * GP_INV_REG];
                y -= g[3] * p[3 * GP_INV_REG];
                x[i] = i == (c0 >> 4) && qc >= 0 && qc < cn ? -gc : y;
            }
        }
        if (own)
#pragma unroll
            for (int i = 0; i < NI; i++)
                if (lane + 16 * i < n) v.inv[(size_t)r * n + lane + 16 * i] = x[i];
        return pg_sync(s);
    }
    // larger: in place in global memory, two barriers a column
    const size_t nn = (size_t)n * n;
    for (size_t e = s.tid; e < nn; e += s.nth) v.inv[e] = 0.0;
    if (!pg_sync(s)) return false;
    for (int t = s.tid; t < n; t += s.nth) {
        v.inv[(size_t)t * n + t] = v.diag[t];
        for (int q = 0; q < v.S; q++) {
            const size_t e = (size_t)q * n + t;
            if (v.col[e] != t) v.inv[(size_t)t * n + v.col[e]] += v.val[e];
        }
    }
    if (!pg_sync(s)) return false;
    for (int c = 0; c < n; c++) {
        if (blockIdx.x == 0) {
            const double d = v.inv[(size_t)c * n + c], inv = 1.0 / (fabs(d) > 1e-300 ? d : 1e-300);
            __syncthreads();
            for (int q = threadIdx.x; q < n; q += blockDim.x)
                v.inv[(size_t)c * n + q] = (q == c ? 1.0 : v.inv[(size_t)c * n + q]) * inv;
        }
        if (!pg_sync(s)) return false;
        for (int t = s.tid >> 5; t < n; t += s.nth >> 5) {       // a warp owns a row
            if (t == c) continue;
            const double f = v.inv[(size_t)t * n + c];
            __syncwarp();
            for (int q = threadIdx.x & 31; q < n; q += 32)
                v.inv[(size_t)t * n + q] = (q == c ? 0.0 : v.inv[(size_t)t * n + q]) - f * v.inv[(size_t)c * n + q];
        }
        if (!pg_sync(s)) return false;
    }
    return true;
}
// operators, pivots and weights of every level (gmg_setup, semiconductor_3d.c:2643-2653): stage
// k builds level k + 1's operator and takes colour k - L of every level L's pivots
__device__ __noinline__ bool gp_setup(const DevP &P, PS &s, const GPArgs &a) {
    const int nl = a.ilu_only ? 1 : a.nl;
    int stages = 0;
    for (int L = 0; L < (nl > 1 ? nl - 1 : nl); L++) stages = max(stages, L + max(a.lev[L].ncolor, 1));
    stages = max(stages, nl - 1);
    for (int k = 0; k < stages; k++) {
        if (k < nl - 1) {
            gp_galerkin(a.lev[k], a.lev[k + 1], k == 0 && a.qsign ? a.lev[0].w : nullptr, s.tid, s.nth);
            if (k + 2 < nl) gp_weights(P, a.lev[k + 1], a.lev[k + 2], k + 1, a.qsign, s.tid, s.nth);
        }
        for (int L = 0; L <= k && L < (nl > 1 ? nl - 1 : nl); L++)
            if (k - L < a.lev[L].ncolor) gp_pivots(a.lev[L], k - L, s.tid, s.nth);
        if (!pg_sync(s)) return false;
    }
    return nl > 1 ? gp_invert(s, a, a.lev[nl - 1]) : true;
}

__global__ void __launch_bounds__(GP_TPB, 1) k_gpersist(const DevP *Ps, GPArgs ga) {
    const DevP &P = Ps[0];
    __shared__ KrylovS sk;
    // the level table in shared memory: after each grid barrier L1 holds nothing, and the
    // passes would otherwise re-read their level descriptors from L2
    __shared__ PGLev lt[GP_MAXL];
    {
        const int words = ga.nl * (int)(sizeof(PGLev) / sizeof(unsigned));
        const unsigned *src = reinterpret_cast<const unsigned *>(ga.lev);
        unsigned *dst = reinterpret_cast<unsigned *>(lt);
        for (int q = threadIdx.x; q < words; q += blockDim.x) dst[q] = src[q];
    }
    GPArgs a = ga;
    a.lev = lt;
    PS s;
    s.g = P.pgrid;
    s.target = 0;
    s.rb = 0;
    s.tid = blockIdx.x * blockDim.x + threadIdx.x;
    s.nth = gridDim.x * blockDim.x;
    s.wait_ns = PG_WAIT_NS;
    s.trace = nullptr;
    s.ntrace = 0;
    s.mode = 1;
    s.onecl = ga.onecl;
    if (threadIdx.x == 0) sk = ga.rec;
    __syncthreads();
    const PGLev &H0 = lt[0];
    const int N = P.N;
    double *x = P.sol;                            // mesh order; everything else in colour order
    double *r = P.wk[0], *rh = P.wk[1], *p = P.wk[2];
    // the system: values, diagonal and row weights in colour order, r = b - A x, its squared
    // norm and rounding floor (semiconductor_3d.c:2244-2268); weights towards level 1
    double acc[3] = {0.0, 0.0, 0.0};
    for (int t = s.tid; t < N; t += s.nth) {
        const int k = H0.node[t];
        const double dg = P.A[0][k], bk = P.rhs[k], dx = dg * x[k];
        double sum = dx, fl = fabs(dx) + fabs(bk);
        for (int q = 0; q < H0.S; q++) {
            const size_t e = (size_t)q * N + t;
            const int se = H0.src[e];
            const double v = se >= 0 ? P.gval[se] : 0.0, tv = v * x[H0.node[H0.col[e]]];
            H0.val[e] = v;
            sum += tv;
            fl += fabs(tv);
        }
        H0.diag[t] = dg;
        H0.w[t] = P.dsc[k];
        const double rk = bk - sum;
        r[t] = rk;
        if (a.kind) { rh[t] = rk; p[t] = rk; }
        // a sweep from zero multiplies what lies in its rows by the zero coupling of their padding
        // slots before it has written them: nothing an earlier solve left there may be a NaN or Inf
        // (tests for the padding in the sweeps instead cost 5 % of a solve)
        (a.kind ? P.wk[4] : P.wk[1])[t] = 0.0;
        if (a.kind) P.wk[5][t] = 0.0;
        acc[0] += rk * rk;
        acc[1] += fl * fl;
    }
    for (int L = 1; L < a.nl - 1; L++)
        for (int t = s.tid; t < lt[L].N; t += s.nth) lt[L].x[t] = 0.0;
    if (a.nl > 1 && !a.ilu_only) gp_weights(P, H0, lt[1], 0, a.qsign, s.tid, s.nth);
    {
        double a2[2] = {acc[0], acc[1]};
        if (!pg_sum<2>(s, a2)) return;
        if (threadIdx.x == 0) {
            if (a.kind) {
                sk.rr = a2[0]; sk.fl = a2[1];
                sk.r0 = sqrt(a2[0]);
                sk.tgt = fmax(a.rtol * sk.r0, a.atol * sqrt(a2[1]));
                sk.rho1 = a2[0]; sk.rbest = sk.r0; sk.stall = 0; sk.it = 0; sk.half = 0;
                sk.active = sk.r0 > sk.tgt ? 1 : 0;
                sk.status = sk.active ? 0 : 1;
            } else {
                sk.active = 1;
            }
        }
        __syncthreads();
    }
    if (sk.active && !gp_setup(P, s, a)) return;
    if (a.kind == 0) {                            // PCG (gpcg), one reduction per iteration (kernels_persist.cu)
        double *z = P.wk[1], *q = P.wk[3], *w = P.wk[4], *zw = P.wk[5];
        p = P.wk[2];
        bool first = true;
        for (;;) {
            if (!gp_vcycle(s, a, r, z, zw)) return;
            double a2[2] = {0.0, 0.0};
            gp_spmv(H0, s, z, [&](int t, double y) {
                w[t] = y;
                a2[0] += r[t] * z[t];
                a2[1] += z[t] * y;
            });
            if (!pg_sum<2>(s, a2)) return;
            if (threadIdx.x == 0) {
                const double rz = a2[0];
                sk.be = 0.0;
                if (first) {
                    sk.rz0 = rz;
                    sk.it = 0;
                    sk.status = rz > 0.0 ? 0 : 2;
                    sk.active = rz > 0.0;
                    sk.pq = a2[1];
                } else if (!(rz > sk.rtol * sk.rtol * sk.rz0)) { sk.active = 0; sk.status = 1; }
                else if (sk.it >= sk.maxit) { sk.active = 0; sk.status = 3; }
                else {
                    sk.be = rz / sk.rz;
                    sk.pq = a2[1] - sk.be * sk.be * sk.pq;
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
            const double al = sk.al, be = sk.be;
            for (int t = s.tid; t < N; t += s.nth) {
                const double pk = first ? z[t] : z[t] + be * p[t], qk = first ? w[t] : w[t] + be * q[t];
                p[t] = pk;
                q[t] = qk;
                x[H0.node[t]] += al * pk;
                r[t] -= al * qk;
            }
            first = false;
            if (!pg_sync(s)) return;
        }
    } else {                                      // BiCGSTAB (gbicgstab)
        double *v = P.wk[3], *ph = P.wk[4], *sh = P.wk[5], *u = P.wk[6];
        // (u serves the V-cycles as the post-smoothing's vector and then holds t = A sh)
        if (threadIdx.x == 0) bicg_next(sk);      // (before the barrier: kernels_persist.cu)
        __syncthreads();
        while (sk.active) {
            double a1[1], a2[2];
            if (sk.pad0) {
                for (int t = s.tid; t < N; t += s.nth) { rh[t] = r[t]; p[t] = r[t]; }
                if (!pg_sync(s)) return;
            }
            if (!gp_vcycle(s, a, p, ph, u)) return;
            a1[0] = 0.0;
            gp_spmv(H0, s, ph, [&](int t, double y) {
                v[t] = y;
                a1[0] += rh[t] * y;
            });
            if (!pg_sum<1>(s, a1)) return;
            if (threadIdx.x == 0) {
                if (fabs(a1[0]) < 1e-300) { sk.active = 0; sk.status = 2; }
                else { sk.rv = a1[0]; sk.al = sk.rho1 / a1[0]; }
            }
            __syncthreads();
            if (!sk.active) break;
            const double al = sk.al;
            a2[0] = a2[1] = 0.0;
            for (int t = s.tid; t < N; t += s.nth) {
                const double y = r[t] - al * v[t];
                r[t] = y;
                a2[0] += y * y;
                a2[1] += rh[t] * y;
            }
            if (!pg_sum<2>(s, a2)) return;
            const double rhs_ = a2[1];
            if (threadIdx.x == 0) {
                sk.ss = a2[0];
                if (sqrt(a2[0]) <= sk.tgt) { sk.half = 1; sk.rr = a2[0]; }
            }
            __syncthreads();
            if (sk.half) {                        // half-step exit: x += al ph
                for (int t = s.tid; t < N; t += s.nth) x[H0.node[t]] += al * ph[t];
                if (threadIdx.x == 0) { sk.active = 0; sk.status = 1; }
                __syncthreads();
                break;
            }
            if (!gp_vcycle(s, a, r, sh, u)) return;
            acc[0] = acc[1] = acc[2] = 0.0;
            gp_spmv(H0, s, sh, [&](int t, double y) {
                u[t] = y;
                acc[0] += y * y;
                acc[1] += r[t] * y;
                acc[2] += rh[t] * y;
            });
            if (!pg_sum<3>(s, acc)) return;
            if (threadIdx.x == 0) {
                sk.tt = acc[0]; sk.ts = acc[1];
                sk.om = acc[0] > 0.0 ? acc[1] / acc[0] : 0.0;
                const double rho = rhs_ - sk.om * acc[2];          // rh . (s - om t)
                sk.be = sk.om != 0.0 ? (rho / sk.rho1) * (sk.al / sk.om) : 0.0;
                sk.rho1 = rho;
            }
            __syncthreads();
            {
                const double om = sk.om, be = sk.be;
                a1[0] = 0.0;
                for (int t = s.tid; t < N; t += s.nth) {
                    x[H0.node[t]] += al * ph[t] + om * sh[t];
                    const double y = r[t] - om * u[t];
                    r[t] = y;
                    p[t] = y + be * (p[t] - om * v[t]);
                    a1[0] += y * y;
                }
            }
            if (!pg_sum<1>(s, a1)) return;
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
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s.g->rec[0] = sk;
        s.g->iters = sk.it;
    }
}

// ---------------------------------------------------------------- host side
namespace {
int g_gp_blocks = 0;               // co-resident blocks of k_gpersist (0: not read yet)
int g_gp_clusters = 0;             // co-resident clusters of GP_CL of them
}

// Tables of the persistent solves from the hierarchy's levels (once per mesh): everything in
// colour-order positions.  Leaves d.g.gptab null when the persistent path cannot serve this
// hierarchy (too many levels or colours, a coarsest level without an inverse, no memory).
void gpersist_build(Inst &d, const std::vector<GpLevelIn> &lv, cudaStream_t st) {
    const int nl = (int)lv.size();
    if (nl > GP_MAXL) return;
    for (const auto &l : lv)
        if (l.ncolor > GP_MAXC) return;
    if (nl > 1 && !d.g.glev[nl - 1].dv.inv) return;
    struct Tab { std::vector<int> col, src, rev, agg, mrp, mem, eptr, elist, dptr, dlist, node; };
    std::vector<Tab> T(nl);
    std::vector<std::vector<int>> pos(nl), eat(nl);      // node -> position; CSR entry -> table entry
    std::vector<PGLev> tab(nl);
    for (int L = 0; L < nl; L++) {
        const GpLevelIn &l = lv[L];
        const int n = l.N;
        const std::vector<int> &rp = *l.rp, &cj = *l.cj, &co = *l.color, &cn = *l.cnodes;
        pos[L].resize(n);
        for (int t = 0; t < n; t++) pos[L][cn[t]] = t;
        int DL = 0, DU = 0;
        for (int k = 0; k < n; k++) {
            int lo = 0;
            for (int e = rp[k]; e < rp[k + 1]; e++) lo += co[cj[e]] < co[k];
            DL = std::max(DL, lo);
            DU = std::max(DU, rp[k + 1] - rp[k] - lo);
        }
        PGLev &p = tab[L];
        p = PGLev{};
        p.N = n; p.DL = DL; p.S = DL + DU; p.ncolor = l.ncolor;
        for (int c = 0; c <= l.ncolor; c++) p.cptr[c] = (*l.cptr)[c];
        Tab &t = T[L];
        t.col.resize((size_t)p.S * n);
        t.src.assign((size_t)p.S * n, -1);
        t.rev.assign((size_t)DL * n, 0);
        eat[L].assign(cj.size(), 0);
        for (int x = 0; x < n; x++) {
            const int k = cn[x];
            int lo = 0, hi = DL;
            for (int e = rp[k]; e < rp[k + 1]; e++) {
                const int q = co[cj[e]] < co[k] ? lo++ : hi++;
                t.col[(size_t)q * n + x] = pos[L][cj[e]];
                t.src[(size_t)q * n + x] = (e - rp[k]) * n + k;      // the mesh's ELL entry
                eat[L][e] = q * n + x;
            }
            for (; lo < DL; lo++) t.col[(size_t)lo * n + x] = x;
            for (; hi < p.S; hi++) t.col[(size_t)hi * n + x] = x;
        }
        for (int k = 0; k < n; k++)
            for (int e = rp[k]; e < rp[k + 1]; e++) {
                const int j = cj[e];
                if (co[j] >= co[k]) continue;
                for (int f = rp[j]; f < rp[j + 1]; f++)
                    if (cj[f] == k) { t.rev[eat[L][e]] = eat[L][f]; break; }
            }
        if (L == 0) t.node = cn;
        // a dimension no slot uses still needs one for the padded reads
    }
    for (int L = 0; L + 1 < nl; L++) {
        const GpLevelIn &l = lv[L], &c = lv[L + 1];
        Tab &t = T[L];
        const int n = l.N, nc = c.N, Sc = tab[L + 1].S;
        t.agg.resize(n);
        for (int x = 0; x < n; x++) t.agg[x] = pos[L + 1][(*l.agg)[(*l.cnodes)[x]]];
        t.mrp.assign(nc + 1, 0);
        for (int x = 0; x < n; x++) t.mrp[t.agg[x] + 1]++;
        for (int I = 0; I < nc; I++) t.mrp[I + 1] += t.mrp[I];
        t.mem.resize(n);
        std::vector<int> at(t.mrp.begin(), t.mrp.end() - 1);
        for (int x = 0; x < n; x++) t.mem[at[t.agg[x]]++] = x;
        t.eptr.assign((size_t)nc * Sc + 1, 0);
        t.dptr.assign(nc + 1, 0);
        auto slot = [&](int e) {                           // fine CSR entry -> coarse row * Sc + slot, -1 inside
            const int ce = (*l.emap)[e];
            if (ce < 0) return -1;
            const int a = eat[L + 1][ce];
            return (a % nc) * Sc + a / nc;
        };
        for (int pass = 0; pass < 2; pass++) {
            std::vector<int> ea, da;
            if (pass) {
                for (size_t q = 0; q + 1 < t.eptr.size(); q++) t.eptr[q + 1] += t.eptr[q];
                for (int I = 0; I < nc; I++) t.dptr[I + 1] += t.dptr[I];
                t.elist.resize(t.eptr.back());
                t.dlist.resize(t.dptr.back());
                ea.assign(t.eptr.begin(), t.eptr.end() - 1);
                da.assign(t.dptr.begin(), t.dptr.end() - 1);
            }
            for (int k = 0; k < n; k++)
                for (int e = (*l.rp)[k]; e < (*l.rp)[k + 1]; e++) {
                    const int q = slot(e), I = t.agg[pos[L][k]];
                    if (q >= 0) {
                        if (pass) t.elist[ea[q]++] = eat[L][e];
                        else t.eptr[q + 1]++;
                    } else if (pass) t.dlist[da[I]++] = eat[L][e];
                    else t.dptr[I + 1]++;
                }
        }
    }
    size_t off = 0;
    auto room = [&](size_t b) { const size_t x = off; off += (b + 255) & ~size_t(255); return x; };
    struct Off { size_t col, src, rev, agg, mrp, mem, eptr, elist, dptr, dlist, node, val, diag, dil, pw, ph, x, b, w; };
    std::vector<Off> O(nl);
    const size_t o_tab = room(sizeof(PGLev) * nl), o_pr = room(sizeof(double) * 2 * 4 * GP_INV_REG);
    for (int L = 0; L < nl; L++) {
        const Tab &t = T[L];
        const size_t n = (size_t)tab[L].N, Sn = (size_t)tab[L].S * n;
        Off &o = O[L];
        o.col = room(t.col.size() * 4); o.src = room(L ? 0 : t.src.size() * 4); o.rev = room(t.rev.size() * 4);
        o.agg = room(t.agg.size() * 4); o.mrp = room(t.mrp.size() * 4); o.mem = room(t.mem.size() * 4);
        o.eptr = room(t.eptr.size() * 4); o.elist = room(t.elist.size() * 4);
        o.dptr = room(t.dptr.size() * 4); o.dlist = room(t.dlist.size() * 4); o.node = room(t.node.size() * 4);
        o.val = room(Sn * 8); o.diag = room(n * 8); o.dil = room(n * 8); o.pw = room(n * 8); o.ph = room(n * 8);
        o.x = room(L ? n * 8 : 0); o.b = room(L ? n * 8 : 0); o.w = room(L ? 0 : n * 8);
    }
    char *blk = nullptr;
    if (cudaMalloc(&blk, off) != cudaSuccess) { cudaGetLastError(); return; }
    bool ok = cudaMemsetAsync(blk, 0, off, st) == cudaSuccess;
    auto up = [&](size_t x, const std::vector<int> &v) {
        if (!v.empty() && cudaMemcpyAsync(blk + x, v.data(), v.size() * 4, cudaMemcpyHostToDevice, st) != cudaSuccess) ok = false;
        return (const int *)(blk + x);
    };
    for (int L = 0; L < nl; L++) {
        const Tab &t = T[L];
        const Off &o = O[L];
        PGLev &p = tab[L];
        p.col = up(o.col, t.col);
        p.src = L ? nullptr : up(o.src, t.src);
        p.rev = up(o.rev, t.rev);
        p.agg = up(o.agg, t.agg); p.mrp = up(o.mrp, t.mrp); p.mem = up(o.mem, t.mem);
        p.eptr = up(o.eptr, t.eptr); p.elist = up(o.elist, t.elist);
        p.dptr = up(o.dptr, t.dptr); p.dlist = up(o.dlist, t.dlist);
        p.node = L ? nullptr : up(o.node, t.node);
        p.val = (double *)(blk + o.val); p.diag = (double *)(blk + o.diag); p.dil = (double *)(blk + o.dil);
        p.pw = (double *)(blk + o.pw); p.ph = (double *)(blk + o.ph);
        p.x = L ? (double *)(blk + o.x) : nullptr;
        p.b = L ? (double *)(blk + o.b) : nullptr;
        p.w = L ? nullptr : (double *)(blk + o.w);
        p.inv = d.g.glev[L].dv.inv;
    }
    if (cudaMemcpyAsync(blk + o_tab, tab.data(), sizeof(PGLev) * nl, cudaMemcpyHostToDevice, st) != cudaSuccess) ok = false;
    if (cudaStreamSynchronize(st) != cudaSuccess) ok = false;
    if (!ok) { cudaGetLastError(); cudaFree(blk); return; }
    d.g.gptab = blk;                               // the table lies at the start of the allocation
    d.g.gprow = blk + o_pr;
}

// Launch the persistent graph solve (kind 0 PCG from the present sol with the stop rule
// r.z <= rtol^2 r0.z0; kind 1 BiCGSTAB with max(rtol r0, atol floor)).  Returns 1 when it
// ran (k holds it, rr, r0), 0 when it does not apply (nothing changed), -1 when a barrier
// wait ran out (the caller restores the start).
int persist_graph(Inst &d, int kind, int maxit, double rtol, double atol, int qsign, bool ilu_only, KrylovS &k) {
    if (!persist_enabled() || !d.g.gptab) return 0;
    const int nl = (int)d.g.glev.size();
    int Ls = nl;
    for (int L = 1; L < nl && Ls == nl; L++)
        if (d.g.glev[L].dv.N <= GP_SMALL) Ls = L;
    if (nl < 2 && !ilu_only) return 0;
    if (!g_gp_blocks) {
        int per = 0, dev = 0, nsm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_gpersist, GP_TPB, 0);
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        cudaLaunchConfig_t q = {};
        q.gridDim = dim3(GP_CL);
        q.blockDim = dim3(GP_TPB);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = GP_CL; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        q.attrs = at;
        q.numAttrs = 1;
        int ncl = 0;
        if (cudaOccupancyMaxActiveClusters(&ncl, k_gpersist, &q) != cudaSuccess) { cudaGetLastError(); ncl = 0; }
        g_gp_clusters = ncl;
        g_gp_blocks = per * nsm;
        cudaGetLastError();
    }
    int nb = g_gp_blocks;
    const int want = (int)((d.N + GP_TPB - 1) / GP_TPB);
    if (want < nb) nb = want < 4 ? 4 : want;
    const int cap = persist_cap(d.pblocks);
    if (cap < nb) nb = cap;
    if (nb < 1) return 0;
    // one cluster of GP_CL blocks, or of what a smaller cap allows
    const int csz = g_gp_clusters > 0 && (nb <= GP_CL || d.N <= (size_t)GP_CLUSTER_N) ? persist_one_cluster(cap) : 0;
    if (csz) nb = csz;
    Ctx c = make_ctx(d);
    KrylovS ks0{};
    ks0.maxit = maxit;
    ks0.rtol = rtol;
    ks0.atol = atol;
    ks0.active = 1;
    PGrid *g = c.h.pgrid;
    cudaMemsetAsync(g, 0, 6 * sizeof(unsigned), c.st);
    GPArgs a{};
    a.lev = reinterpret_cast<const PGLev *>(d.g.gptab);
    a.prow = reinterpret_cast<double *>(d.g.gprow);
    a.nl = nl;
    a.Ls = Ls;
    a.kind = kind;
    a.ilu_only = ilu_only ? 1 : 0;
    a.qsign = qsign;
    a.onecl = csz ? 1 : 0;
    a.alpha = kind ? g_knobs.mg_alpha : g_knobs.mg_alpha_p;
    a.rtol = rtol;
    a.atol = atol;
    a.rec = ks0;
    const DevP *dp = c.dP;
    void *args[] = {(void *)&dp, (void *)&a};
    g_launches++;
    t_launches++;
    if (g_prof_on) prof_begin(PF_PERSIST, c.st);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nb);
    cfg.blockDim = dim3(GP_TPB);
    cfg.stream = c.st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = csz; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = csz ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelExC(&cfg, (const void *)k_gpersist, args);
    if (g_prof_on) prof_end(PF_PERSIST, c.st, 0.0);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    persist_note(nb, csz);
    PGridHead h{};                                // status and closing record in one copy
    const int rc = persist_record(c, g, &h);
    if (rc == 1) k = h.rec[0];
    else
        std::fprintf(stderr, "semisim-b200: persistent graph solve abandoned (%s)\n",
                     h.err == 1 ? "a barrier wait ran out" : "its closing record did not arrive");
    return rc;
}

}  // namespace ss
