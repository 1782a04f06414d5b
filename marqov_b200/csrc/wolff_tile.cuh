// Wolff clusters of hypercubic lattices (2D, 3D) by labelling in bit tiles.
//
// With bond draws keyed by the undirected bond, the Wolff cluster is the
// seed's connected component of the activated bonds between candidates (int8:
// sites in the seed's old state; float: sites whose projection on the
// reflection vector has the seed's sign -- no other site can join).  Three
// launches label the components and flip the seed's:
//   tile_label  a CTA per tile of U units; a unit is a 32-site word of an
//               x-line, held by one thread.  Candidates are a bit per site
//               (warp ballots); the bonds between two candidates are listed
//               per warp and drawn side by side over the lanes, so no lane
//               idles on a bond that needs no draw; bonds active along x
//               join the sites of a word into runs without any union, and
//               the active bonds between units (one per pair of runs where
//               they are adjacent) are united by union-find on 16-bit
//               parents in shared memory.  The tile's candidate and x-bond
//               words and its run labels go to global memory, its local
//               roots enter the global forest;
//   tile_hook   one thread per bond that leaves its tile, united in the
//               global forest of local roots;
//   tile_flip   the local roots of a tile look up whether they hang below the
//               seed's root, the runs follow their local roots, and the
//               sites of the words so marked are flipped and counted.
// What bounds it: the draws -- one Philox block per bond between two
// candidates, about 0.4 bonds per site at the 2D critical point -- and, on
// small lattices, the latency of the dependent steps.
#pragma once
#include "batch.h"
#include "f32_site.cuh"
#include "wolff_int8.cuh"

namespace mqv {

struct CclSeed {
    int64_t rsite;
    int val, newq;  // int8
    float r[3];     // float
    double a;       // float: the seed's projection on r
};

__device__ __forceinline__ int64_t rep_n(const BatchRep& R)
{
    return R.lat_kind == MQV_LATTICE_HYPERCUBIC ? R.st.n : R.csr.n;
}

// Place of a tile and of this thread's unit in it (a 2D tile is one word wide
// and U rows tall; the units of a tile in y and z are powers of two).
template <int U>
struct TileAt {
    int L, Lz;       // side, z extent (1 in 2D)
    int lty, TY, TZ; // units of a tile in y (and its log2) and z
    int tx, ty, tz;  // tile coordinates (words, y tiles, z tiles)
    __device__ __forceinline__ TileAt(const BatchRep& R, int t)
    {
        constexpr int lu = U == 64 ? 6 : U == 128 ? 7 : 8, l3 = tile_ty3(U) == 8 ? 3 : 4;
        const bool d3 = R.st.dim == 3;
        L = R.st.len;
        Lz = d3 ? L : 1;
        lty = d3 ? l3 : lu;
        TY = 1 << lty;
        TZ = d3 ? U >> l3 : 1;
        tx = t % R.tl_nw;
        const int q = t / R.tl_nw;
        tz = d3 ? q / R.tl_ny : 0;
        ty = q - tz * R.tl_ny;
    }
    __device__ __forceinline__ int uy(int u) const { return u & (TY - 1); }
    __device__ __forceinline__ int uz(int u) const { return u >> lty; }
    // x-line of unit u, or -1 beyond the lattice
    __device__ __forceinline__ int row(int u) const
    {
        const int y = (ty << lty) + uy(u), z = tz * TZ + uz(u);
        return (y < L && z < Lz) ? y + L * z : -1;
    }
};

// first site of the run that holds bit b (S: first sites of the runs)
__device__ __forceinline__ int run_start(uint32_t S, int b) { return 31 - __clz(S & (0xFFFFFFFFu >> (31 - b))); }

// union-find on the tile's parents: of two roots the larger id hangs below the
// smaller by an atomic minimum, and a lost race goes on from the parent it
// found instead of from the start
__device__ __forceinline__ int tile_find(volatile int* p, int x)
{
    int px;
    while ((px = p[x]) != x) {
        const int gp = p[px];
        if (gp == px) return px;
        p[x] = gp;
        x = gp;
    }
    return x;
}
__device__ __forceinline__ void tile_unite(int* p, int a, int b)
{
    a = tile_find(p, a);
    b = tile_find(p, b);
    while (a != b) {
        const int lo = min(a, b), hi = max(a, b), old = atomicMin(p + hi, lo);
        if (old == hi) return;
        a = tile_find(p, lo);
        b = tile_find(p, old);
    }
}
// union-find on the global forest of local roots
__device__ __forceinline__ int forest_find(int* __restrict__ p, int x)
{
    while (true) {
        const int px = __ldcg(p + x);
        if (px == x) return x;
        const int gp = __ldcg(p + px);
        if (gp != px) p[x] = gp;  // path halving (races only shorten paths)
        x = gp;
    }
}
__device__ __forceinline__ void forest_unite(int* __restrict__ p, int a, int b)
{
    while (true) {
        a = forest_find(p, a);
        b = forest_find(p, b);
        if (a == b) return;
        if (uf_prio((uint32_t)a) > uf_prio((uint32_t)b)) {
            const int t = a;
            a = b;
            b = t;
        }
        if (atomicCAS(p + a, a, b) == a) return;
    }
}

// activation of the bond (lo, hi) of a float member given both ends'
// projections on the reflection vector
__device__ __forceinline__ bool ccl_active_f32(const BatchRep& R, uint32_t serial, int64_t lo, int64_t hi, double alo,
                                               double ahi)
{
    const double cpl = embed_cpl(R.md.J, alo, ahi);
    return cpl > 0 && !update_accepted(2, cpl, R.md.beta,
                                       lo64(philox((uint32_t)lo, serial, (uint32_t)hi, tag(kWolffBond, R.replica), R.key)));
}
// activation of the bond between candidates i and j
template <bool F32>
__device__ __forceinline__ bool tile_active(const BatchRep& R, const WolffDev& w, Key key, uint32_t tgb,
                                            const float r[3], uint32_t serial, uint32_t i, uint32_t j)
{
    if (F32) {
        const float* s = (const float*)R.s;
        const int64_t n = R.st.n;
        const uint32_t lo = i < j ? i : j, hi = i < j ? j : i;
        return ccl_active_f32(R, serial, lo, hi, embed_proj(R.md.symd, s, n, lo, r[0], r[1], r[2]),
                              embed_proj(R.md.symd, s, n, hi, r[0], r[1], r[2]));
    }
    return wolff_int8_active(w, i, j, serial, tgb, key);
}

template <bool F32>
__device__ __forceinline__ void tile_seed(const BatchRep& R, uint32_t serial, CclSeed& sd)
{
    const uint32_t tgs = tag(kWolffSeed, R.replica);
    if (F32) {
        sd.rsite = embed_seed(R.md, R.st.n, R.key, serial, tgs, sd.r);
        sd.a = embed_proj(R.md.symd, (const float*)R.s, R.st.n, sd.rsite, sd.r[0], sd.r[1], sd.r[2]);
    } else {
        sd.rsite = wolff_int8_seed(R.w, R.st, (const int8_t*)R.s, R.key, serial, tgs, sd.val, sd.newq);
    }
}

// the cluster's serial and its slot in the cluster sizes
__device__ __forceinline__ uint32_t cluster_serial(const BatchRep& R, const BatchCtr* ctr, const ClusterStep& k)
{
    return R.cluster0 + (ctr->e + k.e_off) * (uint32_t)k.ncluster + (uint32_t)k.c + k.serial_add;
}
__device__ __forceinline__ size_t cluster_slot(const BatchCtr* ctr, const ClusterStep& k, int nrep, int r)
{
    const uint32_t slot = ctr->e + k.e_off - ctr->ebase;
    return ((size_t)slot * k.ncluster + k.c) * nrep + r;
}

// (L = 4096, 16.8 M sites at the critical point: 176 us, against 415 for the
// site-by-site kernel in 16 x 16 tiles; L = 1024: 25 against 31 us, with 10
// against 24 us in each of the two launches after it.)
// LPU lanes share a unit: lane l of a warp works on bits [32 / LPU * (l % LPU),
// ...) of unit l / LPU of the warp's 32 / LPU units, so that a lane's serial
// steps over bonds and runs shrink with LPU (latency, on lattices that leave
// the chip half empty) where LPU = 1 keeps the lanes evenest (throughput).
template <bool F32, int U, int LPU>
__global__ void __launch_bounds__(U * LPU, 1280 / (U * LPU))
    tile_label(const BatchRep* __restrict__ reps, const int32_t* __restrict__ tile_prefix,
               const int32_t* __restrict__ tile_rep, CclSeed* __restrict__ seeds, const BatchCtr* __restrict__ ctr,
               ClusterStep step, int32_t* __restrict__ csize, int nrep)
{
    constexpr int NT = U * LPU, UW = 32 / LPU, BITS = 32 / LPU;
    __shared__ __align__(16) int P[U * 32];
    __shared__ unsigned short lists[U * 32];  // a list of bonds per warp
    __shared__ uint32_t sC[U], sB[3][U], sS[U];
    __shared__ CclSeed s_seed;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int u = tid / LPU;  // this lane's unit
    unsigned short* list = lists + warp * (UW * 32);
    // the bonds Q of the warp's units (this lane's part of its unit), listed
    auto list_bonds = [&](uint32_t Q) -> int {
        const int cnt = __popc(Q);
        int pos = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, pos, o);
            if (lane >= o) pos += v;
        }
        const int total = __shfl_sync(0xffffffffu, pos, 31);
        pos -= cnt;
        __syncwarp();  // the list's last readers are done
        while (Q) {
            const int b = __ffs(Q) - 1;
            Q &= Q - 1;
            list[pos++] = (unsigned short)(((lane / LPU) << 5) | b);
        }
        __syncwarp();
        return total;
    };
    const uint32_t part = (LPU == 1 ? 0xFFFFFFFFu : (1u << (BITS & 31)) - 1u) << (BITS * (tid % LPU));
    grid_dep_launch();
    grid_dep_wait();
    const int r = tile_rep[blockIdx.x], t = (int)blockIdx.x - tile_prefix[r];
    const BatchRep& R = reps[r];
    const uint32_t serial = cluster_serial(R, ctr, step);
    const TileAt<U> at(R, t);
    const int dim = R.st.dim, L = at.L;
    const int row = at.row(u), xb = at.tx * 32;
    int* forest = R.tl_forest;
    uint32_t *gcand = R.tl_cand + (int64_t)t * U, *gxb = R.tl_xb + (int64_t)t * U;
    uint4* lab = reinterpret_cast<uint4*>(R.tl_lab + (int64_t)t * (U * 32));
    if (tid == 0) {
        CclSeed sd{};
        tile_seed<F32>(R, serial, sd);
        s_seed = sd;
        if (t == 0) {
            seeds[r] = sd;
            csize[cluster_slot(ctr, step, nrep, r)] = 0;
        }
    }
    if (tid < U) sB[0][tid] = sB[1][tid] = sB[2][tid] = 0u;
#pragma unroll
    for (int k = 0; k < 32 / LPU; ++k) P[k * NT + tid] = k * NT + tid;
    __syncthreads();
    const float rv[3] = {s_seed.r[0], s_seed.r[1], s_seed.r[2]};
    // candidates: the warp's lanes read the 32 sites of one unit after the other
    {
        const int x = xb + lane;
        uint32_t C = 0u;
        if (F32) {
            const double as = s_seed.a;
            const int64_t seed = s_seed.rsite;
#pragma unroll 8
            for (int k = 0; k < UW; ++k) {
                const int rk = __shfl_sync(0xffffffffu, row, k * LPU);
                bool c = false;
                if (rk >= 0 && x < L) {
                    const int64_t i = (int64_t)rk * L + x;
                    const double a = embed_proj(R.md.symd, (const float*)R.s, R.st.n, i, rv[0], rv[1], rv[2]);
                    c = (as > 0 && a > 0) || (as < 0 && a < 0) || i == seed;
                }
                const uint32_t m = __ballot_sync(0xffffffffu, c);
                if (lane == k) C = m;
            }
        } else {
            const int val = s_seed.val;
            const int8_t* s = (const int8_t*)R.s + (R.st.split ? split_addr(0, x, L) : (int64_t)x);
#pragma unroll 8
            for (int k = 0; k < UW; ++k) {
                const int rk = __shfl_sync(0xffffffffu, row, k * LPU);
                const bool c = rk >= 0 && x < L && s[(int64_t)rk * L] == val;
                const uint32_t m = __ballot_sync(0xffffffffu, c);
                if (lane == k) C = m;
            }
        }
        if (lane < UW) {
            sC[warp * UW + lane] = C;
            gcand[warp * UW + lane] = C;
        }
    }
    __syncthreads();
    const uint32_t C = sC[u];
    // the active bonds inside the tile, drawn from the warp's list of bonds
    // between two candidates
    {
        const WolffDev w = R.w;
        const Key key = R.key;
        const uint32_t tgb = tag(kWolffBond, R.replica);
        for (int d = 0; d < dim; ++d) {
            uint32_t Q, step_j;
            if (d == 0) {
                Q = C & (C >> 1);
                step_j = 1u;
            } else if (d == 1) {
                Q = at.uy(u) < at.TY - 1 ? C & sC[u + 1] : 0u;
                step_j = (uint32_t)L;
            } else {
                Q = at.uz(u) < at.TZ - 1 ? C & sC[u + at.TY] : 0u;
                step_j = (uint32_t)L * (uint32_t)L;
            }
            const int total = list_bonds(Q & part);
            for (int k0 = 0; k0 < total; k0 += 32) {
                const int k = k0 + lane;
                const uint32_t id = list[k < total ? k : 0];
                const int rk = __shfl_sync(0xffffffffu, row, (id >> 5) * LPU);
                const uint32_t i = (uint32_t)rk * (uint32_t)L + (uint32_t)xb + (id & 31u);
                if (k < total && tile_active<F32>(R, w, key, tgb, rv, serial, i, i + step_j))
                    atomicOr(&sB[d][warp * UW + (id >> 5)], 1u << (id & 31u));
            }
        }
    }
    __syncthreads();
    // runs, and one union per pair of adjacent runs that active bonds join
    const uint32_t X = sB[0][u], S = C & ~(X << 1);
    if (tid % LPU == 0) {
        sS[u] = S;
        gxb[u] = X;
    }
    __syncthreads();
    // Along y every run first takes the run below its lowest active bond as
    // its parent, by a plain store (parents point to smaller units, so no
    // cycle); only its further bonds, to other runs below, need a union.
    uint32_t more = 0u;
    if (at.uy(u) > 0) {
        const uint32_t Y = sB[1][u - 1], A = X << 1, E = (Y << 1) & A;
        const uint32_t above = E | (((A + E) ^ A) & A);  // sites joined along x to a lower active bond
        for (uint32_t m = Y & ~above & part; m; m &= m - 1) {
            const int b = __ffs(m) - 1;
            P[u * 32 + run_start(S, b)] = (u - 1) * 32 + run_start(sS[u - 1], b);
        }
        // the bond to the left joins the same two runs
        more = Y & above & ~((Y & X & sB[0][u - 1]) << 1) & part;
    }
    __syncthreads();
    for (int d = 1; d < dim; ++d) {
        const int du = d == 1 ? -1 : at.TY;
        if (d == 2) {
            more = sB[2][u];
            if (more) more &= ~((more & X & sB[0][u + du]) << 1) & part;
        }
        const int total = list_bonds(more);
        for (int k = lane; k < total; k += 32) {
            const int id = list[k], ua = warp * UW + (id >> 5), ub = ua + du, b = id & 31;
            tile_unite(P, ua * 32 + run_start(sS[ua], b), ub * 32 + run_start(sS[ub], b));
        }
    }
    __syncthreads();
    const int base = t * (U * 32);
    for (uint32_t m = S & part; m; m &= m - 1) {
        // read-only walks: a parent halved here could overwrite a root written by the run's own thread
        const int x = u * 32 + __ffs(m) - 1;
        int root = x, px;
        while ((px = ((volatile int*)P)[root]) != root) root = px;
        if (root == x) forest[base + x] = base + x;
        else P[x] = root;
    }
    __syncthreads();
#pragma unroll
    for (int k = tid; k < U * 4; k += NT) {
        const int4 p = reinterpret_cast<const int4*>(P)[2 * k], q = reinterpret_cast<const int4*>(P)[2 * k + 1];
        lab[k] = make_uint4((uint32_t)(p.x | (p.y << 16)), (uint32_t)(p.z | (p.w << 16)),
                            (uint32_t)(q.x | (q.y << 16)), (uint32_t)(q.z | (q.w << 16)));
    }
}

template <bool F32, int U, int LPU>
__global__ void __launch_bounds__(U * LPU)
    tile_hook(const BatchRep* __restrict__ reps, const int32_t* __restrict__ tile_prefix,
              const int32_t* __restrict__ tile_rep, const CclSeed* __restrict__ seeds,
              const BatchCtr* __restrict__ ctr, ClusterStep step)
{
    grid_dep_launch();
    grid_dep_wait();
    const int r = tile_rep[blockIdx.x], t = (int)blockIdx.x - tile_prefix[r];
    const BatchRep& R = reps[r];
    const uint32_t serial = cluster_serial(R, ctr, step);
    const TileAt<U> at(R, t);
    const int L = at.L, TY = at.TY, TZ = at.TZ;
    int* forest = R.tl_forest;
    // the tile's last unit row in y and z, the bonds that leave it: one per
    // unit along x, 32 per unit of the y face, 32 per unit of the z face
    const int yl = min(TY - 1, L - 1 - at.ty * TY), zl = min(TZ - 1, at.Lz - 1 - at.tz * TZ);
    const int items = U + 32 * TZ + (R.st.dim == 3 ? 32 * TY : 0);
    const float rv[3] = {F32 ? seeds[r].r[0] : 0.f, F32 ? seeds[r].r[1] : 0.f, F32 ? seeds[r].r[2] : 0.f};
    for (int k0 = 0; k0 < items; k0 += U * LPU) {
        const int k = k0 + (int)threadIdx.x;
        int u = 0, b = 0, t2 = t, u2 = 0, b2 = 0;
        bool live = k < items;
        if (k < U) {
            u = k;
            b = min(31, L - 1 - at.tx * 32);
            t2 = at.tx + 1 < R.tl_nw ? t + 1 : t - at.tx;
            u2 = u;
            b2 = 0;
        } else if (k < U + 32 * TZ) {
            const int q = k - U, z = q >> 5;
            b = b2 = q & 31;
            u = yl + TY * z;
            const int y = at.ty * TY + yl;
            t2 = y + 1 < L ? t + R.tl_nw : t - at.ty * R.tl_nw;
            u2 = TY * z;
            live = z <= zl;
        } else if (live) {
            const int q = k - U - 32 * TZ, y = q >> 5;
            b = b2 = q & 31;
            u = y + TY * zl;
            const int z = at.tz * TZ + zl, plane = R.tl_nw * R.tl_ny;
            t2 = z + 1 < L ? t + plane : t - at.tz * plane;
            u2 = y;
        }
        const int row = at.row(u);
        live = live && row >= 0;
        uint32_t C = 0u, C2 = 0u, X = 0u, X2 = 0u;
        if (live) {
            C = R.tl_cand[(int64_t)t * U + u];
            C2 = R.tl_cand[(int64_t)t2 * U + u2];
            X = R.tl_xb[(int64_t)t * U + u];
            X2 = R.tl_xb[(int64_t)t2 * U + u2];
            live = ((C >> b) & 1u) && ((C2 >> b2) & 1u);
        }
        if (live) {
            const TileAt<U> at2(R, t2);
            const uint32_t i = (uint32_t)row * (uint32_t)L + (uint32_t)(at.tx * 32 + b);
            const uint32_t j = (uint32_t)at2.row(u2) * (uint32_t)L + (uint32_t)(at2.tx * 32 + b2);
            live = tile_active<F32>(R, R.w, R.key, tag(kWolffBond, R.replica), rv, serial, i, j);
        }
        int ra = 0, rb = 0;
        if (live) {
            ra = t * (U * 32) + R.tl_lab[(int64_t)t * (U * 32) + u * 32 + run_start(C & ~(X << 1), b)];
            rb = t2 * (U * 32) + R.tl_lab[(int64_t)t2 * (U * 32) + u2 * 32 + run_start(C2 & ~(X2 << 1), b2)];
        }
        // lanes that join the same two local roots unite them once
        const unsigned long long pair =
            live ? ((unsigned long long)(uint32_t)min(ra, rb) << 32) | (uint32_t)max(ra, rb) : ~0ull;
        const unsigned peers = __match_any_sync(0xffffffffu, pair);
        if (live && ra != rb && (int)(threadIdx.x & 31u) == __ffs(peers) - 1) forest_unite(forest, ra, rb);
    }
}

// global id of the local root of candidate bit b of unit (t, u)
template <int U>
__device__ __forceinline__ int tile_root_of(const BatchRep& R, int t, int u, uint32_t C, int b)
{
    const uint32_t X = R.tl_xb[(int64_t)t * U + u];
    const int start = run_start(C & ~(X << 1), b);
    return t * (U * 32) + (int)R.tl_lab[(int64_t)t * (U * 32) + u * 32 + start];
}

template <bool F32, int U, int LPU>
__global__ void __launch_bounds__(U * LPU)
    tile_flip(const BatchRep* __restrict__ reps, const int32_t* __restrict__ tile_prefix,
              const int32_t* __restrict__ tile_rep, const CclSeed* __restrict__ seeds,
              const BatchCtr* __restrict__ ctr, ClusterStep step, int32_t* __restrict__ csize, int nrep)
{
    constexpr int NT = U * LPU, UW = 32 / LPU, BITS = 32 / LPU;
    __shared__ __align__(16) unsigned short P[U * 32];
    __shared__ uint32_t in[U], hit[U];
    __shared__ int s_root, s_cnt;
    const int tid = threadIdx.x, lane = tid & 31, u = tid / LPU;
    const uint32_t part = (LPU == 1 ? 0xFFFFFFFFu : (1u << (BITS & 31)) - 1u) << (BITS * (tid % LPU));
    grid_dep_launch();
    grid_dep_wait();
    const int r = tile_rep[blockIdx.x], t = (int)blockIdx.x - tile_prefix[r];
    const BatchRep& R = reps[r];
    const CclSeed sd = seeds[r];
    const TileAt<U> at(R, t);
    const int L = at.L, base = t * (U * 32);
    const uint32_t C = R.tl_cand[(int64_t)t * U + u], X = R.tl_xb[(int64_t)t * U + u], S = C & ~(X << 1);
    const uint4* lab = reinterpret_cast<const uint4*>(R.tl_lab + base);
#pragma unroll
    for (int k = tid; k < U * 4; k += NT) reinterpret_cast<uint4*>(P)[k] = lab[k];
    if (tid < U) in[tid] = hit[tid] = 0u;
    const int* forest = R.tl_forest;
    auto walk = [&](int x) {
        int p;
        while ((p = __ldcg(forest + x)) != x) x = p;
        return x;
    };
    if (tid == NT - 1) {
        // the seed's root
        const uint32_t i = (uint32_t)sd.rsite, rw = R.st.lg >= 0 ? i >> R.st.lg : R.st.divlen(i);
        const int x = (int)(i - rw * (uint32_t)L);
        const int z = at.Lz > 1 ? (int)(R.st.lg >= 0 ? rw >> R.st.lg : R.st.divlen(rw)) : 0, y = (int)rw - z * L;
        const int st = (x >> 5) + R.tl_nw * ((y >> at.lty) + R.tl_ny * (z / at.TZ)),
                  su = at.uy(y) + at.TY * (z % at.TZ);
        s_root = walk(tile_root_of<U>(R, st, su, R.tl_cand[(int64_t)st * U + su], x & 31));
        s_cnt = 0;
    }
    __syncthreads();
    const int root = s_root;
    // the forest above each local root of this lane's part of its unit
    // (four first steps in flight: most local roots are roots of the forest)
    uint32_t f = 0u, mine = 0u;
    for (uint32_t m = S & part; m; m &= m - 1) {
        const int b = __ffs(m) - 1;
        if (P[u * 32 + b] == u * 32 + b) mine |= 1u << b;
    }
    while (mine) {
        int b[4], p[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            b[k] = __ffs(mine) - 1;
            mine &= mine - 1;
            p[k] = b[k] >= 0 ? __ldcg(forest + base + u * 32 + b[k]) : -1;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (b[k] >= 0 && (p[k] == base + u * 32 + b[k] ? p[k] : walk(p[k])) == root) f |= 1u << b[k];
    }
    if (f) atomicOr(&in[u], f);
    __syncthreads();
    for (uint32_t m = S & part & ~f; m; m &= m - 1) {
        const int b = __ffs(m) - 1, l = P[u * 32 + b];
        if ((in[l >> 5] >> (l & 31)) & 1u) f |= 1u << b;
    }
    if (LPU > 1) {
        if (f) atomicOr(&hit[u], f);
        __syncwarp();
        f = hit[u];
    }
    // the runs of the marked first sites: a carry ripples up each run's bonds
    {
        const uint32_t A = X << 1, E = (f << 1) & A;
        f |= E | (((A + E) ^ A) & A);
        f &= C;
    }
    const int cnt = __reduce_add_sync(0xffffffffu, tid % LPU == 0 ? __popc(f) : 0);
    if (lane == 0 && cnt) atomicAdd(&s_cnt, cnt);
    const int row = at.row(u), x = at.tx * 32 + lane;
    if (cnt) {
        int8_t* s8 = (int8_t*)R.s + (F32 ? 0 : R.st.split ? split_addr(0, x, L) : (int64_t)x);
        for (int k = 0; k < UW; ++k) {
            const uint32_t fk = __shfl_sync(0xffffffffu, f, k * LPU);
            const int rk = __shfl_sync(0xffffffffu, row, k * LPU);
            if (!((fk >> lane) & 1u)) continue;
            if (F32) embed_reflect(R.md.symd, (float*)R.s, R.st.n, (int64_t)rk * L + x, sd.r[0], sd.r[1], sd.r[2]);
            else s8[(int64_t)rk * L] = (int8_t)sd.newq;
        }
    }
    __syncthreads();
    if (tid == 0 && s_cnt) atomicAdd(csize + cluster_slot(ctr, step, nrep, r), s_cnt);
}

}  // namespace mqv
