// Wolff clusters by connected-component labelling, site by site, for CSR
// graphs and one- and four-dimensional lattices (2D and 3D lattices are
// labelled in bit tiles, wolff_tile.cuh).
//
// With bond draws keyed by the undirected bond (lower id, cluster serial,
// upper id), the Wolff cluster is the seed's connected component of the
// activated bonds, whatever the visiting order.  A breadth-first growth from
// one CTA needs one step per level of the cluster; this variant labels every
// component of the activated-bond graph of every member in a fixed number of
// whole-lattice passes -- lock-free union-find: each undirected bond once,
// roots hooked by compare-and-swap in a fixed pseudo-random order (uf_prio),
// paths halved on the way -- and flips the
// seed's component:
//   ccl_seed      one thread per member: seed site, old/new state or the
//                 reflection vector (the same substream draws as the BFS);
//   ccl_local     per CTA of 256 consecutive sites: candidates (int8: state
//                 equal to the seed's old state; float: every site)
//                 get labels, and activated bonds with both ends in the CTA's
//                 sites are united in shared memory first; each candidate's
//                 label becomes its local root, non-candidates get -1;
//   ccl_hook      the other activated bonds between candidates are united;
//   ccl_halve     every candidate's path to its root halved;
//   ccl_flip      members of the seed's component (read-only walks to the
//                 roots) are flipped / reflected and counted into the cluster
//                 size.
// The label array is the member's BFS queue (n int32); the visited bitmap is
// not touched.
#pragma once
#include "batch.h"
#include "f32_site.cuh"
#include "wolff_int8.cuh"
#include "wolff_tile.cuh"

namespace mqv {

// member and local site of flattened site g
__device__ __forceinline__ int ccl_member(int64_t g, const int64_t* __restrict__ prefix,
                                          const int32_t* __restrict__ block_rep, int64_t& i)
{
    int r = block_rep[blockIdx.x];
    while (g >= prefix[r + 1]) ++r;
    i = g - prefix[r];
    return r;
}

__device__ __forceinline__ int ccl_find(int* __restrict__ p, int x)
{
    while (true) {
        const int px = __ldcg(p + x);
        if (px == x) return x;
        const int gp = __ldcg(p + px);
        if (gp != px) p[x] = gp;  // path halving (races only shorten paths)
        x = gp;
    }
}

__device__ __forceinline__ void ccl_unite(int* __restrict__ p, int a, int b)
{
    while (true) {
        a = ccl_find(p, a);
        b = ccl_find(p, b);
        if (a == b) return;
        if (uf_prio((uint32_t)a) > uf_prio((uint32_t)b)) {  // the root of lower priority hangs below
            const int t = a;
            a = b;
            b = t;
        }
        if (atomicCAS(p + a, a, b) == a) return;
    }
}

template <bool F32>
__global__ void ccl_seed(const BatchRep* __restrict__ reps, const BatchCtr* __restrict__ ctr, ClusterStep step,
                         CclSeed* __restrict__ seeds, int32_t* __restrict__ csize, int nrep)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrep) return;
    const BatchRep& R = reps[r];
    if (R.resident || R.tl_tiles) return;  // clusters grown by batch_resident / labelled in tiles
    const uint32_t serial = cluster_serial(R, ctr, step);
    const uint32_t tgs = tag(kWolffSeed, R.replica);
    CclSeed sd{};
    if (F32) {
        sd.rsite = embed_seed(R.md, rep_n(R), R.key, serial, tgs, sd.r);
    } else if (R.lat_kind == MQV_LATTICE_HYPERCUBIC) {
        sd.rsite = wolff_int8_seed(R.w, R.st, (const int8_t*)R.s, R.key, serial, tgs, sd.val, sd.newq);
    } else {
        sd.rsite = wolff_int8_seed(R.w, R.csr, (const int8_t*)R.s, R.key, serial, tgs, sd.val, sd.newq);
    }
    seeds[r] = sd;
    csize[cluster_slot(ctr, step, nrep, r)] = 0;
}

// activation of the bond (i, j) between two candidate sites of member R, on
// the bond's keyed draw (the breadth-first growth's rule)
template <bool F32>
__device__ __forceinline__ bool ccl_active(const BatchRep& R, const CclSeed& sd, uint32_t serial, int64_t i, int64_t j)
{
    const uint32_t tgb = tag(kWolffBond, R.replica);
    if (F32) {
        const int64_t lo = i < j ? i : j, hi = i < j ? j : i;
        const float* s = (const float*)R.s;
        const int64_t n = rep_sites(R);
        const double cpl = embed_cpl(R.md.J, embed_proj(R.md.symd, s, n, lo, sd.r[0], sd.r[1], sd.r[2]),
                                     embed_proj(R.md.symd, s, n, hi, sd.r[0], sd.r[1], sd.r[2]));
        return cpl > 0 &&
               !update_accepted(2, cpl, R.md.beta, lo64(philox((uint32_t)lo, serial, (uint32_t)hi, tgb, R.key)));
    }
    return wolff_int8_active(R.w, (uint32_t)i, (uint32_t)j, serial, tgb, R.key);
}

// the forward bonds (i, j) of site i, each undirected bond once: +x, +y, ...
// on stencils, j > i on CSR graphs
template <class F>
__device__ __forceinline__ void ccl_forward_bonds(const BatchRep& R, int64_t i, F&& f)
{
    if (R.lat_kind == MQV_LATTICE_HYPERCUBIC) {
        for (int d = 0; d < R.st.dim; ++d) f(R.st.nbr(i, 2 * d));
    } else {
        for (int t = R.csr.rp[i]; t < R.csr.rp[i + 1]; ++t) {
            const int64_t j = R.csr.ci[t];
            if (j > i) f(j);
        }
    }
}

// union-find on the CTA's shared labels (the same scheme as ccl_find /
// ccl_unite on shared memory)
__device__ __forceinline__ int ccl_lfind(volatile int* p, int x)
{
    while (true) {
        const int px = p[x];
        if (px == x) return x;
        const int gp = p[px];
        if (gp != px) p[x] = gp;
        x = gp;
    }
}
__device__ __forceinline__ void ccl_lunite(volatile int* p, int a, int b)
{
    while (true) {
        a = ccl_lfind(p, a);
        b = ccl_lfind(p, b);
        if (a == b) return;
        if (uf_prio((uint32_t)a) > uf_prio((uint32_t)b)) {  // the root of lower priority hangs below
            const int t = a;
            a = b;
            b = t;
        }
        if (atomicCAS((int*)p + a, a, b) == a) return;
    }
}

// flattened site g and g2 in the same CTA block of kBatchMetroThreads sites
__device__ __forceinline__ bool ccl_same_block(int64_t g, int64_t g2)
{
    return g / kBatchMetroThreads == g2 / kBatchMetroThreads;
}

template <bool F32>
__global__ void __launch_bounds__(kBatchMetroThreads)
    ccl_local(const BatchRep* __restrict__ reps, const int64_t* __restrict__ prefix,
              const int32_t* __restrict__ block_rep, int64_t total, const CclSeed* __restrict__ seeds,
              const BatchCtr* __restrict__ ctr, ClusterStep step)
{
    __shared__ int slab[kBatchMetroThreads];
    const int64_t base = (int64_t)blockIdx.x * kBatchMetroThreads;
    const int64_t g = base + threadIdx.x;
    int r = 0;
    int64_t i = 0;  // this thread's site
    bool cand = false;
    if (g < total) {
        r = ccl_member(g, prefix, block_rep, i);
        const BatchRep& R = reps[r];
        cand = true;
        if (!F32) {
            const int64_t a = R.lat_kind == MQV_LATTICE_HYPERCUBIC ? R.st.addr(i) : i;
            cand = ((const int8_t*)R.s)[a] == seeds[r].val;
        }
    }
    slab[threadIdx.x] = cand ? (int)threadIdx.x : -1;
    __syncthreads();
    if (cand) {
        const BatchRep& R = reps[r];
        const uint32_t serial = cluster_serial(R, ctr, step);
        const CclSeed sd = seeds[r];
        volatile int* vl = slab;
        const int64_t off = prefix[r];
        ccl_forward_bonds(R, i, [&](int64_t j) {
            if (!ccl_same_block(g, off + j)) return;
            const int k = (int)(off + j - base);
            if (vl[k] >= 0 && ccl_active<F32>(R, sd, serial, i, j)) ccl_lunite(vl, (int)threadIdx.x, k);
        });
    }
    __syncthreads();
    if (cand) ccl_lfind(slab, (int)threadIdx.x);  // paths halved side by side first
    __syncthreads();
    if (g < total) {
        int lab = -1;
        if (cand) {
            // read-only walk to the local root (same member: bonds join only its sites)
            int x = (int)threadIdx.x, px;
            while ((px = ((volatile int*)slab)[x]) != x) x = px;
            lab = (int)(base + x - prefix[r]);
        }
        reps[r].queue[i] = lab;
    }
}

template <bool F32>
__global__ void ccl_hook(const BatchRep* __restrict__ reps, const int64_t* __restrict__ prefix,
                         const int32_t* __restrict__ block_rep, int64_t total, const CclSeed* __restrict__ seeds,
                         const BatchCtr* __restrict__ ctr, ClusterStep step)
{
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    int64_t i;
    const int r = ccl_member(g, prefix, block_rep, i);
    const BatchRep& R = reps[r];
    int* lab = R.queue;
    if (__ldcg(lab + i) < 0) return;
    const uint32_t serial = cluster_serial(R, ctr, step);
    const CclSeed sd = seeds[r];
    const int64_t off = prefix[r];
    // bonds within the CTA block were united by ccl_local
    ccl_forward_bonds(R, i, [&](int64_t j) {
        if (ccl_same_block(g, off + j) || __ldcg(lab + j) < 0) return;
        if (ccl_active<F32>(R, sd, serial, i, j)) ccl_unite(lab, (int)i, (int)j);
    });
}

// Every candidate's path halved, all side by side (a write only ever points
// a site to an ancestor, so the forest stays valid while others walk it), so
// that ccl_flip's walks are short.
static __global__ void ccl_halve(const BatchRep* __restrict__ reps, const int64_t* __restrict__ prefix,
                                 const int32_t* __restrict__ block_rep, int64_t total)
{
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    int64_t i;
    const int r = ccl_member(g, prefix, block_rep, i);
    int* lab = reps[r].queue;
    if (__ldcg(lab + i) < 0) return;
    ccl_find(lab, (int)i);
}

template <bool F32>
__global__ void ccl_flip(const BatchRep* __restrict__ reps, const int64_t* __restrict__ prefix,
                         const int32_t* __restrict__ block_rep, int64_t total, const CclSeed* __restrict__ seeds,
                         const BatchCtr* __restrict__ ctr, ClusterStep step, int32_t* __restrict__ csize, int nrep)
{
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool in = false;
    int r = 0;
    if (g < total) {
        int64_t i;
        r = ccl_member(g, prefix, block_rep, i);
        const BatchRep& R = reps[r];
        const CclSeed& sd = seeds[r];
        // read-only walks to the roots (short after ccl_halve)
        const int* lab = R.queue;
        int root = __ldcg(lab + sd.rsite), x = __ldcg(lab + i);
        if (root >= 0 && x >= 0) {
            int p;
            while ((p = __ldcg(lab + root)) != root) root = p;
            while ((p = __ldcg(lab + x)) != x) x = p;
            in = x == root;
        }
        if (in) {
            if (F32) {
                embed_reflect(R.md.symd, (float*)R.s, rep_sites(R), i, sd.r[0], sd.r[1], sd.r[2]);
            } else {
                const int64_t a = R.lat_kind == MQV_LATTICE_HYPERCUBIC ? R.st.addr(i) : i;
                ((int8_t*)R.s)[a] = (int8_t)sd.newq;
            }
        }
    }
    // count per member: lanes of one member aggregate their adds
    const unsigned lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(0xffffffffu, r);
    const unsigned cnt = __popc(__ballot_sync(0xffffffffu, in) & peers);
    if (cnt && lane == (unsigned)(__ffs(peers) - 1)) {
        atomicAdd(csize + cluster_slot(ctr, step, nrep, r), (int)cnt);
    }
}

}  // namespace mqv
