// Anderson acceleration (Walker-Ni) of the Gummel map on the 3N state
// x = (psi, phi_n, phi_p) (semiconductor_3d.c:3709-3757): FP32 difference history,
// FP64 Gram matrix and normal equations, masked mixing.
#include "device_common.cuh"
#include "prof.h"
#include "solver_ctx.h"

namespace ss {

static inline dim3 grid3(const Ctx &c) {
    int b = (3 * c.maxN + TPB - 1) / TPB;
    if (b > c.grid_cap) b = c.grid_cap;
    return dim3(b < 1 ? 1 : b, c.ninst);
}

// carrier `hole` matters at node k: > 1e-6 of n + p + |Nd - Na| (semiconductor_3d.c:3696-3700)
__device__ __forceinline__ bool aa_sig(const DevP &P, int k, int hole) {
    const uint32_t f = P.flags[k];
    if (fl_kind(f) != K_SEMI || fl_fix(f)) return false;
    const double c = hole ? P.p[k] : P.n[k];
    return c > 1e-6 * (P.n[k] + P.p[k] + fabs(P.Nd[k] - P.Na[k]));
}
__device__ __forceinline__ void blk(const DevP &P, int b, const double *&x, double *&g) {
    x = b == 0 ? P.xk : (b == 1 ? P.qn0 : P.qp0);
    g = b == 0 ? P.phi : (b == 1 ? P.phin : P.phip);
}

// One pass over the state for everything before the mix: f = masked (g - x); with a stored
// previous f (m > 0) the new history column s, dF[s] = f - f_old and dG[s] = g - g_old (float),
// the Gram row of dF[s] and the right-hand side dF[i] . f over the m columns; then f and g
// stored.  The last block to finish adds the partial sums (a warp per sum) and its first warp
// solves the regularised normal equations.  What bounds it: m history columns of 4 bytes and
// ~70 bytes of state an entry; as four passes it read the columns twice and the state three
// times, and the normal equations were solved by one thread out of local memory (FinFET of
// 214,000 nodes: 174 us a Gummel iteration, the mix included, now 89 us; 1.9M nodes: 517 and 323 us).
constexpr int AA_NS = 2 * AA_MAX;                         // sums: Gram row, right-hand side
static_assert(AA_NS <= RED_AA, "partial records too small");
__global__ void __launch_bounds__(TPB) k_aa_pass(const DevP *__restrict__ Ps, int s, int m) {
    const DevP &P = Ps[blockIdx.y];
    const int N = P.N, L = 3 * N;
    double acc[AA_NS];
#pragma unroll
    for (int i = 0; i < AA_NS; i++) acc[i] = 0.0;
    float *dF = P.aaF + (size_t)s * L, *dG = P.aaG + (size_t)s * L;
    SS_GRID_LOOP(q, L) {
        const int b = q / N, k = q - b * N;
        const double *x; double *g;
        blk(P, b, x, g);
        const double gk = g[k], xk = x[k];
        float h[AA_MAX];
#pragma unroll
        for (int i = 0; i < AA_MAX; i++) h[i] = i < m && i != s ? P.aaF[(size_t)i * L + q] : 0.f;
        const double f = (b == 0 || aa_sig(P, k, b - 1)) ? gk - xk : 0.0;
        if (m) {
            const float df = (float)(f - P.aaf[q]);
            dF[q] = df;
            dG[q] = (float)(gk - P.aag[q]);
#pragma unroll
            for (int i = 0; i < AA_MAX; i++) {
                const double a = (double)(i == s ? df : h[i]);
                acc[i] += a * (double)df;
                acc[AA_MAX + i] += a * f;
            }
        }
        P.aaf[q] = f;
        P.aag[q] = gk;
    }
    if (!m) return;
    __shared__ double tot[AA_NS], A[AA_MAX][AA_MAX + 1];
    __shared__ bool is_last;
    block_sum<AA_NS>(acc);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < AA_NS; i++) P.part[blockIdx.x * RED_AA + i] = acc[i];
        __threadfence();
        is_last = atomicAdd(P.ticket + 6, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x >> 5; i < AA_NS; i += TPB / 32) {   // in block order: lanes stride the blocks
        double v = 0.0;
        for (int b = lane; b < (int)gridDim.x; b += 32) v += __ldcg(P.part + b * RED_AA + i);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) tot[i] = v;
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    if (lane == 0) *(P.ticket + 6) = 0u;
    if (lane < m) {
        P.gram[lane * AA_MAX + s] = tot[lane];
        P.gram[s * AA_MAX + lane] = tot[lane];
    }
    __syncwarp();
    // lane r holds row r of the normal equations; Gauss-Jordan with partial pivoting
    double tr = 0.0;
    for (int i = 0; i < m; i++) tr += i == s ? tot[s] : P.gram[i * AA_MAX + i];
    if (lane < m) {
        for (int j = 0; j < m; j++)
            A[lane][j] = lane == s ? tot[j] : (j == s ? tot[lane] : P.gram[lane * AA_MAX + j]);
        A[lane][lane] += 1e-9 * tr + 1e-300;
        A[lane][m] = tot[AA_MAX + lane];
    }
    __syncwarp();
    for (int c = 0; c < m; c++) {
        double mx = lane >= c && lane < m ? fabs(A[lane][c]) : -1.0;
        int p = lane;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {                        // rows lie in lanes 0 .. 11
            const double y = __shfl_xor_sync(0xffffffffu, mx, o);
            const int r = __shfl_xor_sync(0xffffffffu, p, o);
            if (y > mx || (y == mx && r < p)) { mx = y; p = r; }
        }
        p = __shfl_sync(0xffffffffu, p, 0);
        if (p < c) p = c;                                        // (no comparable entry: NaN)
        if (p != c && lane <= m) {
            const double t = A[c][lane];
            A[c][lane] = A[p][lane];
            A[p][lane] = t;
        }
        __syncwarp();
        if (lane < m && lane != c) {
            const double f = A[lane][c] / A[c][c];
            for (int q = c; q <= m; q++) A[lane][q] -= f * A[c][q];
        }
        __syncwarp();
    }
    const double gam = lane < m ? A[lane][m] / A[lane][lane] : 0.0;
    if (lane < m) P.aagam[lane] = gam;
    const bool ok = __all_sync(0xffffffffu, gam == gam);
    if (lane == 0) P.res[R_AUX] = ok ? 1.0 : 0.0;
}
// g -= sum gam_i dG[i] where the node takes part (psi off contacts, phi_n/p where significant)
__global__ void k_aa_mix(const DevP *__restrict__ Ps, int m) {
    const DevP &P = Ps[blockIdx.y];
    if (P.res[R_AUX] == 0.0) return;                 // NaN coefficients: keep the Picard step
    const int N = P.N, L = 3 * N;
    double gam[AA_MAX];
    for (int i = 0; i < m; i++) gam[i] = P.aagam[i];
    SS_GRID_LOOP(q, L) {
        const int b = q / N, k = q - b * N;
        const uint32_t f = P.flags[k];
        if (b == 0 ? fl_con(f) != 0 : fl_fix(f)) continue;
        if (b > 0 && !aa_sig(P, k, b - 1)) continue;
        const double *x; double *g;
        blk(P, b, x, g);
        double s = g[k];
        for (int i = 0; i < m; i++) s -= gam[i] * (double)P.aaG[(size_t)i * L + q];
        g[k] = s;
    }
}

void aa_pass(const Ctx &c, int slot, int m) {
    SS_LAUNCH(PF_AA, 3 * c.maxN, k_aa_pass, grid3(c), TPB, c.st, c.dP, slot, m);
    if (m) SS_LAUNCH(PF_AA, 3 * c.maxN, k_aa_mix, grid3(c), TPB, c.st, c.dP, m);
}

}  // namespace ss
