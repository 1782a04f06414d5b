// Runs of joined sites in 32-site words, and forests of them in shared
// memory: the pieces that the bit-plane cluster kernels share (wolff_tile.cuh,
// bits_emcs.cu).
#pragma once
#include <cstdint>

namespace mqv {

// the closure of S along a word through the bonds X (bit b: sites b and b + 1)
// towards higher bits, for S made of first sites of runs: a carry ripples up
// each run
__device__ __forceinline__ uint32_t run_fill(uint32_t S, uint32_t X)
{
    const uint32_t A = X << 1, E = (S << 1) & A;
    return S | E | (((A + E) ^ A) & A);
}
// the sites joined along the word to a lower site of Y
__device__ __forceinline__ uint32_t run_above(uint32_t Y, uint32_t X)
{
    const uint32_t A = X << 1, E = (Y << 1) & A;
    return E | (((A + E) ^ A) & A);
}
// bit i of r at the i-th set bit of m
__device__ __forceinline__ uint32_t bit_deposit(uint32_t r, uint32_t m)
{
    uint32_t out = 0u;
    for (; m; m &= m - 1, r >>= 1)
        if (r & 1u) out |= m & (0u - m);
    return out;
}
// 32 bits of a bit string from bit `pos` on (one word past the end is read)
__device__ __forceinline__ uint32_t bit_string(const uint32_t* w, int pos)
{
    return __funnelshift_r(w[pos >> 5], w[(pos >> 5) + 1], (uint32_t)pos & 31u);
}
// inclusive sum over the lanes
__device__ __forceinline__ int warp_prefix(int v, int lane)
{
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, v, s);
        if (lane >= s) v += o;
    }
    return v;
}
// the or over groups of n lanes (n a power of two)
__device__ __forceinline__ uint32_t group_or(uint32_t v, int n)
{
    for (int s = 1; s < n; s <<= 1) v |= __shfl_xor_sync(0xffffffffu, v, s);
    return v;
}

// Flatten the forest P[0 .. n): every node jumps to its parent's parent, one
// jump per node and pass, all side by side, until every parent is a root (a
// chain of k parents takes about log2 k passes).  Nodes are written by their
// own thread alone.
__device__ __forceinline__ void forest_jump(int* P, int n, int tid, int nt)
{
    volatile int* vp = P;
    bool moved;
    do {
        moved = false;
        for (int k = tid; k < n; k += 4 * nt) {
            int p[4], q[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) p[h] = k + h * nt < n ? vp[k + h * nt] : 0;
#pragma unroll
            for (int h = 0; h < 4; ++h) q[h] = vp[p[h]];
#pragma unroll
            for (int h = 0; h < 4; ++h)
                if (k + h * nt < n && q[h] != p[h]) {
                    vp[k + h * nt] = q[h];
                    moved = true;
                }
        }
    } while (moved);
}
// Join the trees of a and b: the larger node hangs below the smaller by an
// atomic minimum; where it hung below another one before, that one and the
// smaller are joined next.  Parents only ever decrease, so this ends, and no
// tie of the forest is lost.
__device__ __forceinline__ void forest_join(int* P, int a, int b)
{
    a = *(volatile int*)(P + a);
    b = *(volatile int*)(P + b);
    while (a != b) {
        const int lo = min(a, b), hi = max(a, b), old = atomicMin(P + hi, lo);
        if (old == hi) return;
        a = lo;
        b = old;
    }
}

}  // namespace mqv
