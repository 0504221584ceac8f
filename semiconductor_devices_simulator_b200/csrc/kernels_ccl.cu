// Floating majority-carrier blocks of a continuity solve (semiconductor_3d.c:3159-3228).
// A connected region where carrier c is the quasi-neutral majority and that no carrier
// contact reaches is rescaled uniformly, c -> lambda c, so that its global balance
// (net outflow + recombination inside = 0) holds; Newton in ln(lambda) per block.
//
// The reference finds the blocks by a breadth-first search.  Here the components are
// labelled on the device by union-find (ccl_common.cuh) in one merging pass, the anchoring
// test and the block sums are per-node kernels adding into per-block exact accumulators
// (exact_sum.cuh), so that the sums, and the rescaled solution, do not depend on the order of
// the threads.  What bounds it is launches and the wait for the block count, not memory: four
// short kernels and one wait per call (576,000 nodes: 107 us of kernels; min-label propagation by line
// sweeps until nothing changed took 305 us in ~15 launches, and a wait for every turn).
#include <cmath>
#include <cstdio>
#include <vector>

#include "ccl_common.cuh"
#include "device_common.cuh"
#include "exact_sum.cuh"
#include "prof.h"
#include "solver_ctx.h"

namespace ss {

constexpr int FF_MAX_BLOCKS = 1024;

__device__ __forceinline__ bool ff_maj(const DevP &P, int k, int hole) {
    const uint32_t f = P.flags[k];
    if (fl_kind(f) != K_SEMI || fl_con(f)) return false;
    const double s = P.sc[k], c = s * P.sol[k];
    const double oth = hole ? P.n[k] : P.p[k];
    const double hd = 0.5 * dnet_ion(P, k);
    const MatD &m = P.mats[fl_mat(f)];
    return c >= oth && c >= hd && s >= hd && c > 10.0 * niK(P, m, k);
}

// majority nodes start as the first node of their run inside a warp along x (runs of
// consecutive majority nodes of one row), the others as -1
__global__ void k_ff_init(const DevP *__restrict__ Ps, int hole, int *count) {
    const DevP &P = Ps[blockIdx.y];
    const int lane = threadIdx.x & 31, nw = (P.N + 31) & ~31;
    if (blockIdx.x == 0 && threadIdx.x == 0) *count = 0;
    SS_GRID_LOOP(k, nw) {                             // whole warps
        const bool in = k < P.N, maj = in && ff_maj(P, k, hole);
        const bool head = !maj || P.gcol || k % P.Nx == 0;      // (graph nodes are no rows)
        const unsigned m = __ballot_sync(0xffffffffu, maj), h = __ballot_sync(0xffffffffu, head);
        if (in) {
            // the run starts after the last non-majority lane, or at the last row start, below or here
            const unsigned below = (2u << lane) - 1u;
            const unsigned starts = ((h & m) | (m & ~(m << 1))) & below;
            P.ccl[k] = maj ? k - lane + (31 - __clz(starts)) : -1;
            P.cclaux[k] = 0;
        }
    }
}
// join every majority node with its lower neighbours; a link along y or z is left out where
// the previous node along x has the same one (the two rows' runs are already joined there)
__global__ void k_ff_merge(const DevP *__restrict__ Ps) {
    const DevP &P = Ps[blockIdx.y];
    int *lab = P.ccl;
    const int Nx = P.Nx, NxNy = P.Nx * P.Ny;
    SS_GRID_LOOP(k, P.N) {
        if (lab[k] < 0) continue;
        const Node a = unidx(k, Nx, P.Ny);
        const bool left = a.i > 0 && lab[k - 1] >= 0;
        if (left && (k & 31) == 0) uf_union(lab, k, k - 1);      // a run cut at a warp's edge
        if (a.j > 0 && lab[k - Nx] >= 0 && !(left && lab[k - Nx - 1] >= 0)) uf_union(lab, k, k - Nx);
        if (a.l > 0 && lab[k - NxNy] >= 0 && !(left && lab[k - NxNy - 1] >= 0)) uf_union(lab, k, k - NxNy);
    }
}
// every node gets its component's root; a block touching a semiconductor contact node is
// anchored
__global__ void k_ff_anchor(const DevP *__restrict__ Ps) {
    const DevP &P = Ps[blockIdx.y];
    SS_GRID_LOOP(k, P.N) {
        if (P.ccl[k] < 0) continue;
        const int lb = uf_find(P.ccl, k);
        P.ccl[k] = lb;
        const Node a = unidx(k, P.Nx, P.Ny);
        for (int dir = 0; dir < 6; dir++) {
            int kb; double h, ar;
            if (!nbr(P, a, k, dir, kb, h, ar)) continue;
            const uint32_t fb = P.flags[kb];
            if (fl_kind(fb) == K_SEMI && fl_con(fb)) { P.cclaux[lb] = 1; break; }
        }
    }
}
// list the unanchored roots; cclaux[root] = 2 + block index
__global__ void k_ff_roots(const DevP *__restrict__ Ps, int *count, int *roots) {
    const DevP &P = Ps[blockIdx.y];
    SS_GRID_LOOP(k, P.N) {
        if (P.ccl[k] != k || P.cclaux[k] != 0) continue;
        const int b = atomicAdd(count, 1);
        if (b < FF_MAX_BLOCKS) { roots[b] = k; P.cclaux[k] = 2 + b; }
        else P.cclaux[k] = 1;          // beyond the table: left as it is
    }
}
__device__ __forceinline__ int ff_block(const DevP &P, int k) {
    const int lb = P.ccl[k];
    if (lb < 0) return -1;
    const int a = P.cclaux[lb];
    return a >= 2 ? a - 2 : -1;
}
// boundary balance of every block: Aout = sum self s_k u_k, Bin = sum nb c_b
__global__ void k_ff_boundary(const DevP *__restrict__ Ps, int hole, unsigned long long *Aout,
                              unsigned long long *Bin) {
    const DevP &P = Ps[blockIdx.y];
    SS_GRID_LOOP(k, P.N) {
        const int b = ff_block(P, k);
        if (b < 0) continue;
        const Node a = unidx(k, P.Nx, P.Ny);
        const uint32_t f = P.flags[k];
        const MatD &m = P.mats[fl_mat(f)];
        const double VT = m.VT, lk = hole ? lnvK(P, m, k) : lncK(P, m, k);
        const double ck = P.sc[k] * P.sol[k];
        double ao = 0.0, bi = 0.0;
        for (int dir = 0; dir < 6; dir++) {
            int kb; double h, ar;
            if (!nbr(P, a, k, dir, kb, h, ar)) continue;
            const uint32_t fb = P.flags[kb];
            if (fl_kind(fb) != K_SEMI || P.ccl[kb] == P.ccl[k]) continue;
            const MatD &mb = P.mats[fl_mat(fb)];
            const double lb = hole ? lnvK(P, mb, kb) : lncK(P, mb, kb);
            const double D = (P.phi[kb] - P.phi[k]) / VT + (hole ? -(lb - lk) : (lb - lk));
            const int kl = k < kb ? k : kb;
            const double g = ar * P.fmu[(hole ? 3 : 0) + (dir >> 1)][kl] * VT / h;
            const double self = hole ? g * bern(D) : g * bern(-D), nb = hole ? g * bern(-D) : g * bern(D);
            const double cb = fl_con(fb) ? (hole ? P.p[kb] : P.n[kb]) : P.sc[kb] * P.sol[kb];
            ao += self * ck;
            bi += nb * cb;
        }
        xs_add(Aout + (size_t)b * XS_WORDS, ao);
        xs_add(Bin + (size_t)b * XS_WORDS, bi);
    }
}
// recombination of every block at the trial scale lambda_b (null: 1)
__global__ void k_ff_recomb(const DevP *__restrict__ Ps, int hole, const double *lam, unsigned long long *G,
                            unsigned long long *dG) {
    const DevP &P = Ps[blockIdx.y];
    SS_GRID_LOOP(k, P.N) {
        const int b = ff_block(P, k);
        if (b < 0) continue;
        const Node a = unidx(k, P.Nx, P.Ny);
        const MatD &m = P.mats[fl_mat(P.flags[k])];
        const double c = (lam ? lam[b] : 1.0) * P.sc[k] * P.sol[k];
        const double oth = hole ? P.n[k] : P.p[k];
        double R, dRn, dRp;
        recombK(P, m, k, hole ? oth : c, hole ? c : oth, R, dRn, dRp);
        const double vol = P.Lx[a.i] * P.Ly[a.j] * P.Lz[a.l];
        double g = vol * R, dg = vol * (hole ? dRp : dRn) * c;
        if (P.tk) { g += P.tk[k] * c - P.tg[k]; dg += P.tk[k] * c; }   // metal-contact exchange
        if (P.gii) g -= P.gii[k];                                        // impact-ionisation pairs
        xs_add(G + (size_t)b * XS_WORDS, g);
        xs_add(dG + (size_t)b * XS_WORDS, dg);
    }
}
// One Newton step of every block's balance l A - B + G(l) = 0 in s = ln l, a thread a block (one
// CTA): the totals of the boundary sums (first step) and of the recombination sums, the step
// (at most 2), the next trial l, the scale the block gets if it stops here, and the sums cleared
// for the next step.  flag[0]: blocks still moving, flag[1]: blocks rescaled.  On the device so
// that the host waits once a step: with the totals read back and l sent up it waited four times
// a balance (batched resolve of six 36,864-node MOSFETs 74.3 -> 71.4 ms, 576,000-node resolve
// 123.3 -> 122.1).
struct FfState {
    double *A, *B, *lam, *fix, *s, *act;
};
__global__ void __launch_bounds__(TPB) k_ff_newton(unsigned long long *acc, size_t aw, int nb, int first, FfState f, int *flag) {
    __shared__ int cnt[2];
    if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        unsigned long long *const a = acc + (size_t)b * XS_WORDS;
        if (first) {
            f.A[b] = xs_value(a);
            f.B[b] = xs_value(a + aw);
        }
        const double G = xs_value(a + 2 * aw), dG = xs_value(a + 3 * aw);
        for (int q = 0; q < XS_WORDS; q++) a[2 * aw + q] = a[3 * aw + q] = 0;
        const double l = first ? 1.0 : f.lam[b];
        double s = first ? 0.0 : f.s[b];
        bool act = first || f.act[b] != 0.0;
        if (act) {
            const double Gv = l * f.A[b] - f.B[b] + G, dGv = l * f.A[b] + dG;
            if (!(dGv > 0.)) act = false;
            else {
                double ds = -Gv / dGv;
                if (ds > 2.) ds = 2.;
                else if (ds < -2.) ds = -2.;
                s += ds;
                if (fabs(ds) < 1e-13) act = false;
            }
        }
        const double e = exp(s);
        const bool moved = s == s && fabs(s) > 1e-15 && fabs(s) < 200.;
        f.s[b] = s;
        f.act[b] = act ? 1.0 : 0.0;
        f.lam[b] = e;
        f.fix[b] = moved ? e : 1.0;
        if (act) atomicAdd(&cnt[0], 1);
        if (moved) atomicAdd(&cnt[1], 1);
    }
    __syncthreads();
    if (threadIdx.x < 2) flag[threadIdx.x] = cnt[threadIdx.x];
}
__global__ void k_ff_apply(const DevP *__restrict__ Ps, const double *scale) {
    const DevP &P = Ps[blockIdx.y];
    SS_GRID_LOOP(k, P.N) {
        const int b = ff_block(P, k);
        if (b < 0) continue;
        P.sol[k] *= scale[b];
    }
}

int float_fix(Inst &d, int hole) {
    Ctx c = make_ctx(d);
    const dim3 g(c.nodes_blocks(), 1);
    double *const g_ffbuf = d.g.h.ffbuf;
    int *const g_ffint = d.g.h.ffint;
    int *count = g_ffint + 1, *roots = g_ffint + 16;
    SS_LAUNCH(PF_CCL, d.N, k_ff_init, g, TPB, c.st, c.dP, hole, count);
    if (d.unstr) {
        ff_label_g(d);                                        // over the graph's edges, anchors
    } else {
        SS_LAUNCH(PF_CCL, d.N, k_ff_merge, g, TPB, c.st, c.dP);
        SS_LAUNCH(PF_CCL, d.N, k_ff_anchor, g, TPB, c.st, c.dP);
    }
    SS_LAUNCH(PF_CCL, d.N, k_ff_roots, g, TPB, c.st, c.dP, count, roots);
    int *const hp = reinterpret_cast<int *>(d.g.pin);
    cudaMemcpyAsync(hp, count, sizeof(int), cudaMemcpyDeviceToHost, c.st);
    cudaStreamSynchronize(c.st);
    int nb = hp[0];
    if (nb <= 0) return 0;
    if (nb > FF_MAX_BLOCKS) nb = FF_MAX_BLOCKS;
    const FfState f{g_ffbuf, g_ffbuf + FF_MAX_BLOCKS, g_ffbuf + 2 * FF_MAX_BLOCKS, g_ffbuf + 3 * FF_MAX_BLOCKS,
                    g_ffbuf + 4 * FF_MAX_BLOCKS, g_ffbuf + 5 * FF_MAX_BLOCKS};
    int *const flag = g_ffint + 8;
    unsigned long long *const acc = d.g.h.ffacc;           // [sum][block][XS_WORDS]
    const size_t aw = (size_t)FF_MAX_BLOCKS * XS_WORDS;
    cudaMemset2DAsync(acc, aw * sizeof(unsigned long long), 0, sizeof(unsigned long long) * nb * XS_WORDS, 4, c.st);
    if (d.unstr) ff_boundary_g(d, hole, acc, acc + aw);
    else SS_LAUNCH(PF_CCL, d.N, k_ff_boundary, g, TPB, c.st, c.dP, hole, acc, acc + aw);
    int nfix = 0;
    for (int it = 0; it < 60; it++) {
        SS_LAUNCH(PF_CCL, d.N, k_ff_recomb, g, TPB, c.st, c.dP, hole, it ? f.lam : nullptr, acc + 2 * aw, acc + 3 * aw);
        SS_LAUNCH(PF_CCL, nb, k_ff_newton, dim3(1), nb <= 32 ? 32 : TPB, c.st, acc, aw, nb, it == 0, f, flag);
        cudaMemcpyAsync(hp, flag, 2 * sizeof(int), cudaMemcpyDeviceToHost, c.st);
        cudaStreamSynchronize(c.st);
        nfix = hp[1];
        if (!hp[0]) break;
    }
    SS_LAUNCH(PF_CCL, d.N, k_ff_apply, g, TPB, c.st, c.dP, f.fix);
    if (d.verbose > 2) std::fprintf(stderr, "    float_fix(%c): %d blocks, %d rescaled\n", hole ? 'p' : 'n', nb, nfix);
    return nfix;
}

}  // namespace ss
