// Union-find over int32 parents in device memory: the larger root is hooked
// under the smaller, so the final root is the smallest member, whatever the
// order of the unions.  Safe for concurrent unions.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace rtr {

__device__ __forceinline__ int32_t uf_find(int32_t* p, int32_t x)
{
    while (true) {
        const int32_t px = p[x];
        if (px == x) return x;
        const int32_t ppx = p[px];
        if (ppx != px) atomicCAS(&p[x], px, ppx);
        x = px;
    }
}

__device__ __forceinline__ void uf_unite(int32_t* p, int32_t a, int32_t b)
{
    while (true) {
        a = uf_find(p, a);
        b = uf_find(p, b);
        if (a == b) return;
        if (a > b) {
            const int32_t t = a;
            a = b;
            b = t;
        }
        const int32_t old = atomicCAS(&p[b], b, a);
        if (old == b) return;
        b = old;
    }
}

}  // namespace rtr
