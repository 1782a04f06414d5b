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
//               they are adjacent) join the runs' trees in shared memory:
//               the first of a run by a plain store, the others in rounds of
//               hooking and flattening.  The tile's candidate and x-bond
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
// Float bonds are screened in FP32 (embed_active) and a bond that leaves its tile
// finds its far site without dividing: 32 phi^4 chains of 64^3 139 -> 120 us
// (label), 70 -> 59 (hook), 54 (flip) of a cluster.
#pragma once
#include "batch.h"
#include "f32_site.cuh"
#include "runs.cuh"
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

// Embedded Wolff: the bond of coupling cpl > 0 is active when its word does not
// accept (update_accepted<2>).  The acceptance 2^(2 log2(e) (-beta cpl)) in FP32
// is within 1e-5 of the rule's cut; a word that comes no nearer than 1e-4 of it
// (and 1e-6, for the words' own rounding) is decided there, the others exactly.
__device__ __forceinline__ bool embed_active(double cpl, double beta, uint64_t word)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"((float)MQV_DMUL(-beta, cpl) * 2.8853900817779268f));
    const float u = (float)(uint32_t)(word >> 40) * 5.9604644775390625e-8f;
    if (u > y * 1.0001f + 1e-6f) return true;
    if (u + 1e-6f < y * 0.9999f) return false;
    return !update_accepted(2, cpl, beta, word);
}

// what the activation of a member's bonds depends on
struct TileBonds {
    WolffDev w;             // int8
    const float* s;         // float
    int64_t n;
    int symd;
    double J, beta;
    float r[3];
    uint32_t serial, tgb;
    __device__ __forceinline__ TileBonds(const BatchRep& R, const float rv[3], uint32_t serial_)
        : w(R.w), s((const float*)R.s), n(R.st.n), symd(R.md.symd), J(R.md.J), beta(R.md.beta), r{rv[0], rv[1], rv[2]},
          serial(serial_), tgb(tag(kWolffBond, R.replica))
    {
    }
};

// activation of the bond between candidates i and j
template <bool F32, class K>
__device__ __forceinline__ bool tile_active(const TileBonds& B, const K& key, uint32_t i, uint32_t j)
{
    if (F32) {
        const uint32_t lo = i < j ? i : j, hi = i < j ? j : i;
        const double cpl = embed_cpl(B.J, embed_proj(B.symd, B.s, B.n, lo, B.r[0], B.r[1], B.r[2]),
                                     embed_proj(B.symd, B.s, B.n, hi, B.r[0], B.r[1], B.r[2]));
        return cpl > 0 && embed_active(cpl, B.beta, lo64(philox(lo, B.serial, hi, B.tgb, key)));
    }
    return wolff_int8_active(B.w, i, j, B.serial, B.tgb, key);
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

// LPU lanes share a unit: lane l of a warp works on bits [32 / LPU * (l % LPU),
// ...) of unit l / LPU of the warp's 32 / LPU units, so that the steps over the
// bits of a unit shrink with LPU (latency, on lattices that leave the chip
// half empty) where LPU = 1 pays the per-warp steps once per 32 units
// (throughput).
template <bool F32, int U, int LPU>
__global__ void __launch_bounds__(U * LPU, 1280 / (U * LPU))
    tile_label(const BatchRep* __restrict__ reps, const int32_t* __restrict__ tile_prefix,
               const int32_t* __restrict__ tile_rep, CclSeed* __restrict__ seeds, const BatchCtr* __restrict__ ctr,
               ClusterStep step, int32_t* __restrict__ csize, int nrep)
{
    constexpr int NT = U * LPU, UW = 32 / LPU, BITS = 32 / LPU, NW = NT / 32;
    constexpr int DIRS = U == 64 ? 3 : 1;          // directions in one bond list
    constexpr int LIST = UW * 32 * DIRS;           // bond list entries of a warp
    constexpr int EDGES = U * 16;                  // edges between runs (the rest is found again in the planes)
    constexpr int RES = LIST / 32 + 3;             // outcome words of a warp's list
    constexpr int PN = U * 32 > NW * RES ? U * 32 : NW * RES;
    __shared__ __align__(16) int P[PN];            // parents of the runs (before: the outcomes)
    __shared__ uint32_t edge[NW * LIST / 2 > EDGES ? NW * LIST / 2 : EDGES];  // edges (before: the bond lists)
    __shared__ uint32_t sC[U], sB[3][U], sS[U];
    __shared__ int sR[U], s_warp[NW], s_nedge;
    __shared__ CclSeed s_seed;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int u = tid / LPU;  // this lane's unit
    const uint32_t part = (LPU == 1 ? 0xFFFFFFFFu : (1u << (BITS & 31)) - 1u) << (BITS * (tid % LPU));
    grid_dep_launch();
    grid_dep_wait();
    const int r = tile_rep[blockIdx.x], t = (int)blockIdx.x - tile_prefix[r];
    const BatchRep& R = reps[r];
    const uint32_t serial = cluster_serial(R, ctr, step);
    const TileAt<U> at(R, t);
    const int dim = R.st.dim, L = at.L;
    const int row = at.row(u), xb = at.tx * 32, base = t * (U * 32);
    int* forest = R.tl_forest + base;
    unsigned short* lab = R.tl_lab + base;
    uint32_t *gcand = R.tl_cand + (int64_t)t * U, *gxb = R.tl_xb + (int64_t)t * U, *gbase = R.tl_base + (int64_t)t * U;
    if (tid == 0) {
        CclSeed sd{};
        tile_seed<F32>(R, serial, sd);
        s_seed = sd;
        s_nedge = 0;
        if (t == 0) {
            seeds[r] = sd;
            csize[cluster_slot(ctr, step, nrep, r)] = 0;
        }
    }
    if (tid < U) sB[0][tid] = sB[1][tid] = sB[2][tid] = 0u;
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
    const int uy = at.uy(u), uz = at.uz(u);
    // The active bonds inside the tile: the bonds between two candidates are
    // listed per warp and drawn side by side over the lanes; the outcomes come
    // back as a bit string in the list's order.
    {
        const TileBonds bonds(R, rv, serial);
        const RoundKeys key(R.key);
        unsigned short* list = reinterpret_cast<unsigned short*>(edge) + warp * LIST;
        uint32_t* res = reinterpret_cast<uint32_t*>(P) + warp * RES;
        const int first_site = row * L + xb;
        for (int d0 = 0; d0 < dim; d0 += DIRS) {
            uint32_t Q[3] = {0u, 0u, 0u};
            if (d0 == 0) Q[0] = C & (C >> 1) & part;
            if (DIRS == 3 || d0 == 1) Q[1] = uy < at.TY - 1 ? C & sC[u + 1] & part : 0u;
            if ((DIRS == 3 || d0 == 2) && dim == 3) Q[2] = uz < at.TZ - 1 ? C & sC[u + at.TY] & part : 0u;
            const int cnt = __popc(Q[0]) + __popc(Q[1]) + __popc(Q[2]);
            int pos = warp_prefix(cnt, lane);
            const int total = __shfl_sync(0xffffffffu, pos, 31), from = pos -= cnt;
            __syncwarp();  // the list's last readers are done
#pragma unroll
            for (int d = 0; d < 3; ++d)
                for (uint32_t m = Q[d]; m; m &= m - 1)
                    list[pos++] = (unsigned short)((d << 10) | ((lane / LPU) << 5) | (__ffs(m) - 1));
            __syncwarp();
            for (int k0 = 0; k0 < total; k0 += 64) {
                uint32_t i[2], j[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k = k0 + 32 * h + lane;
                    const uint32_t id = list[k < total ? k : 0];
                    i[h] = (uint32_t)__shfl_sync(0xffffffffu, first_site, ((id >> 5) & 31u) * LPU) + (id & 31u);
                    const uint32_t d = id >> 10;
                    j[h] = i[h] + (d == 0 ? 1u : d == 1 ? (uint32_t)L : (uint32_t)L * (uint32_t)L);
                }
                const bool a0 = tile_active<F32>(bonds, key, i[0], j[0]);
                const bool a1 = tile_active<F32>(bonds, key, i[1], j[1]);
                const uint32_t r0 = __ballot_sync(0xffffffffu, a0), r1 = __ballot_sync(0xffffffffu, a1);
                if (lane == 0) {
                    res[k0 >> 5] = r0;
                    res[(k0 >> 5) + 1] = r1;
                }
            }
            __syncwarp();
            int at_bit = from;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (DIRS == 1 && d != d0) continue;
                const uint32_t B = Q[d] ? bit_deposit(bit_string(res, at_bit), Q[d]) : 0u;
                at_bit += __popc(Q[d]);
                const uint32_t all = group_or(B, LPU);
                if (tid % LPU == 0) sB[d][u] = all;
            }
        }
    }
    // Runs: the bonds along x join the sites of a unit.  They are numbered
    // through the tile (sR: first run of every unit), so that the steps below
    // take one run or edge per thread.
    __syncthreads();
    const uint32_t X = sB[0][u], S = C & ~(X << 1);
    if (tid % LPU == 0) {
        sS[u] = S;
        gxb[u] = X;
    }
    __syncthreads();
    {
        const int cnt = tid < U ? __popc(sS[tid]) : 0, pos = warp_prefix(cnt, lane);
        if (lane == 31) s_warp[warp] = pos;
        __syncthreads();
        int before = 0;
#pragma unroll
        for (int k = 0; k < U / 32; ++k) before += k < warp ? s_warp[k] : 0;
        if (tid < U) {
            sR[tid] = before + pos - cnt;
            gbase[tid] = (uint32_t)sR[tid];
        }
    }
    __syncthreads();
    const int nrun = sR[U - 1] + __popc(sS[U - 1]);
    for (int k = tid; k < nrun; k += NT) P[k] = k;
    __syncthreads();
    auto run_of = [&](int v, int b) { return sR[v] + __popc(sS[v] & (0xFFFFFFFFu >> (31 - b))) - 1; };
    // Along y every run first takes the run below its lowest active bond as
    // its parent, by a plain store; the further bonds between runs, one per
    // pair where they are adjacent, are the edges left, listed.
    auto edges_z = [&](int v, uint32_t Xv) -> uint32_t {
        const uint32_t Z = sB[2][v];
        return Z ? Z & ~((Z & Xv & sB[0][v + at.TY]) << 1) : 0u;
    };
    {
        uint32_t ey = 0u, ez = 0u;
        if (uy > 0) {
            const uint32_t Y = sB[1][u - 1], above = run_above(Y, X);
            for (uint32_t m = Y & ~above & part; m; m &= m - 1) {
                const int b = __ffs(m) - 1;
                P[run_of(u, b)] = run_of(u - 1, b);
            }
            ey = Y & above & ~((Y & X & sB[0][u - 1]) << 1) & part;
        }
        if (dim == 3) ez = edges_z(u, X) & part;
        const int cnt = __popc(ey) + __popc(ez), pos = warp_prefix(cnt, lane);
        int slot = 0;
        if (lane == 31 && pos) slot = atomicAdd(&s_nedge, pos);
        slot = __shfl_sync(0xffffffffu, slot, 31) + pos - cnt;
        for (; ey; ey &= ey - 1, ++slot)
            if (slot < EDGES) edge[slot] = (uint32_t)run_of(u, __ffs(ey) - 1) | ((uint32_t)run_of(u - 1, __ffs(ey) - 1) << 16);
        for (; ez; ez &= ez - 1, ++slot)
            if (slot < EDGES)
                edge[slot] = (uint32_t)run_of(u, __ffs(ez) - 1) | ((uint32_t)run_of(u + at.TY, __ffs(ez) - 1) << 16);
    }
    __syncthreads();
    const int nedge = min(s_nedge, EDGES);
    forest_jump(P, nrun, tid, NT);
    __syncthreads();
    for (int k = tid; k < nedge; k += NT) forest_join(P, (int)(edge[k] & 0xFFFFu), (int)(edge[k] >> 16));
    if (s_nedge > EDGES && tid < U) {  // more than the list holds: once more from the planes
        if (at.uy(tid) < at.TY - 1)
            for (uint32_t m = sB[1][tid]; m; m &= m - 1)
                forest_join(P, run_of(tid, __ffs(m) - 1), run_of(tid + 1, __ffs(m) - 1));
        if (dim == 3)
            for (uint32_t m = sB[2][tid]; m; m &= m - 1)
                forest_join(P, run_of(tid, __ffs(m) - 1), run_of(tid + at.TY, __ffs(m) - 1));
    }
    __syncthreads();
    forest_jump(P, nrun, tid, NT);
    __syncthreads();
    for (int k = tid; k < nrun; k += NT) {
        const int p = P[k];
        lab[k] = (unsigned short)p;
        if (p == k) forest[k] = base + k;
    }
}

// global id of the local root of candidate bit b of unit (t, u), whose words
// are C and X
template <int U>
__device__ __forceinline__ int tile_root_of(const BatchRep& R, int t, int u, uint32_t C, uint32_t X, int b)
{
    const uint32_t S = C & ~(X << 1);
    const int run = (int)R.tl_base[(int64_t)t * U + u] + __popc(S & (0xFFFFFFFFu >> (31 - b))) - 1;
    return t * (U * 32) + (int)R.tl_lab[(int64_t)t * (U * 32) + run];
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
    const TileBonds bonds(R, rv, serial);
    for (int k0 = 0; k0 < items; k0 += U * LPU) {
        const int k = k0 + (int)threadIdx.x;
        // unit and bit of the site, tile, unit and bit of its neighbour, and the
        // neighbour's x-line less the site's
        int u = 0, b = 0, t2 = t, u2 = 0, b2 = 0, drow = 0;
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
            drow = y + 1 < L ? 1 : 1 - L;
            u2 = TY * z;
            live = z <= zl;
        } else if (live) {
            const int q = k - U - 32 * TZ, y = q >> 5;
            b = b2 = q & 31;
            u = y + TY * zl;
            const int z = at.tz * TZ + zl, plane = R.tl_nw * R.tl_ny;
            t2 = z + 1 < L ? t + plane : t - at.tz * plane;
            drow = z + 1 < L ? L : L - L * L;
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
            const int x = at.tx * 32 + b, x2 = k >= U ? x : x + 1 < L ? x + 1 : 0;
            live = tile_active<F32>(bonds, R.key, (uint32_t)(row * L + x), (uint32_t)((row + drow) * L + x2));
        }
        int ra = 0, rb = 0;
        if (live) {
            ra = tile_root_of<U>(R, t, u, C, X, b);
            rb = tile_root_of<U>(R, t2, u2, C2, X2, b2);
        }
        // lanes that join the same two local roots unite them once
        const unsigned long long pair =
            live ? ((unsigned long long)(uint32_t)min(ra, rb) << 32) | (uint32_t)max(ra, rb) : ~0ull;
        const unsigned peers = __match_any_sync(0xffffffffu, pair);
        if (live && ra != rb && (int)(threadIdx.x & 31u) == __ffs(peers) - 1) forest_unite(forest, ra, rb);
    }
}

template <bool F32, int U, int LPU>
__global__ void __launch_bounds__(U * LPU)
    tile_flip(const BatchRep* __restrict__ reps, const int32_t* __restrict__ tile_prefix,
              const int32_t* __restrict__ tile_rep, const CclSeed* __restrict__ seeds,
              const BatchCtr* __restrict__ ctr, ClusterStep step, int32_t* __restrict__ csize, int nrep)
{
    constexpr int NT = U * LPU, UW = 32 / LPU, BITS = 32 / LPU;
    __shared__ unsigned short lab[U * 32];
    __shared__ uint32_t in[U + 1], hit[U + 1];  // a bit per run, in order
    __shared__ int s_root, s_cnt, s_nrun;
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
    const int run0 = (int)R.tl_base[(int64_t)t * U + u];
    const int* forest = R.tl_forest;
    auto walk = [&](int x) {
        int p;
        while ((p = __ldcg(forest + x)) != x) x = p;
        return x;
    };
    if (tid == NT - 1) {  // a lane of the tile's last unit
        s_nrun = run0 + __popc(S);
        s_cnt = 0;
    }
    __syncthreads();
    const int nrun = s_nrun;
#pragma unroll 4
    for (int k = tid; k < nrun; k += NT) lab[k] = R.tl_lab[base + k];
    if (tid == 0) {
        // the seed's root
        const uint32_t i = (uint32_t)sd.rsite, rw = R.st.lg >= 0 ? i >> R.st.lg : R.st.divlen(i);
        const int x = (int)(i - rw * (uint32_t)L);
        const int z = at.Lz > 1 ? (int)(R.st.lg >= 0 ? rw >> R.st.lg : R.st.divlen(rw)) : 0, y = (int)rw - z * L;
        const int st = (x >> 5) + R.tl_nw * ((y >> at.lty) + R.tl_ny * (z / at.TZ)),
                  su = at.uy(y) + at.TY * (z % at.TZ);
        s_root = walk(tile_root_of<U>(R, st, su, R.tl_cand[(int64_t)st * U + su], R.tl_xb[(int64_t)st * U + su], x & 31));
    }
    __syncthreads();
    const int root = s_root;
    // The forest above each local root.  A walk is a chain of dependent loads:
    // a lane takes those of four runs side by side.
    for (int k0 = tid - lane; k0 < nrun; k0 += 4 * NT) {
        int x[4];  // -1: not a local root
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + j * NT + lane;
            x[j] = k < nrun && lab[k] == k ? base + k : -1;
        }
        bool open;
        do {
            int p[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) p[j] = x[j] >= 0 ? __ldcg(forest + x[j]) : -1;
            open = false;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                open = open || p[j] != x[j];
                x[j] = p[j];
            }
        } while (open);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (k0 + j * NT >= nrun) break;
            const uint32_t m = __ballot_sync(0xffffffffu, x[j] == root);
            if (lane == 0) in[(k0 + j * NT) >> 5] = m;
        }
    }
    __syncthreads();
    // every run follows its local root
    for (int k0 = tid - lane; k0 < nrun; k0 += NT) {
        const int k = k0 + lane, l = k < nrun ? lab[k] : 0;
        const uint32_t m = __ballot_sync(0xffffffffu, k < nrun && ((in[l >> 5] >> (l & 31)) & 1u));
        if (lane == 0) hit[k0 >> 5] = m;
    }
    __syncthreads();
    // ... and the words' sites their runs
    const uint32_t mine = S & part;
    uint32_t f = mine ? bit_deposit(bit_string(hit, run0 + __popc(S & (part - 1u) & ~part)), mine) : 0u;
    f = group_or(f, LPU);
    if (f) f = run_fill(f, X);
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
