// Connected components by union-find on a parent array (tensor and graph meshes): every
// labelled node points at a node of its component with a smaller or equal index, a root at
// itself, unlabelled nodes hold -1.  Merging hooks the larger root under the smaller one by
// atomicMin, so a component's root ends as its smallest node - the label that min-label
// propagation ends with, in one pass instead of one per turn of the shape.
#pragma once
#include <cuda_runtime.h>

namespace ss {

// root of node k; every step goes to a smaller index, so it ends
__device__ __forceinline__ int uf_find(const int *lab, int k) {
    for (;;) {
        const int p = *reinterpret_cast<const volatile int *>(lab + k);
        if (p == k) return k;
        k = p;
    }
}
// join the components of a and b.  A hook that finds its root already hooked elsewhere goes
// on from there; the larger of the two indices falls in every round, so it ends
__device__ __forceinline__ void uf_union(int *lab, int a, int b) {
    for (;;) {
        a = uf_find(lab, a);
        b = uf_find(lab, b);
        if (a == b) return;
        if (a < b) { const int t = a; a = b; b = t; }
        const int old = atomicMin(lab + a, b);
        if (old == a) return;
        a = old;
    }
}

}  // namespace ss
