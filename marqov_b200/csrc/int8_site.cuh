// Device building blocks of the int8 models shared by the per-handle kernels
// (metropolis_int8.cu) and the batched kernels (batch.cu): the per-site
// Metropolis update, the checkerboard site map, the observable accumulation
// and its finalisation.
#pragma once
#include "engine.h"

namespace mqv {

// ---------------------------------------------------------------------------
// generic per-site update (Metropolis<H,L>::move, src/libmarqov/metropolis.h:88-126)

// `cuts`: the u53 cut of every dE the model can produce (host table
// int8_cut_table), D the bound of a neighbourhood sum that it was made for; the decision equals
// update_accepted<1>(dE, beta, word) on the site's acceptance word.  `sub`:
// the site's sublattice (checkerboard colour) where the lattice has a
// termselector.  Lanes with live == false touch no memory.
template <class Lat, class SP>
__device__ __forceinline__ void int8_site(const ModelDev& m, const Lat& lat, SP s, int64_t i,
                                          Key key, uint32_t sweep, uint32_t replica,
                                          const unsigned long long* __restrict__ cuts, int D, bool live, int sub = 0,
                                          const uint4* tab = nullptr, uint32_t run0 = 0)
{
    int64_t ai = 0;
    int nw = 0;
    uint64_t cut = 0;
    if (live) {
        SubStream rng(key, (uint32_t)i, sweep, tag(kMetro, replica));
        ai = lat.addr(i);
        const int old = s[ai];
        const int deg = lat.degree(i);
        int k;
        if (m.kind == MQV_MODEL_POTTS) {
            // Initializer<Potts<Q>>::newsv (src/hamiltonian/Potts.h:170-177) and
            // PottsInteraction::diff (src/hamiltonian/Potts.h:86-107)
            nw = (int)mod_small(rng.next(), (uint32_t)m.q);
            int eo = 0, en = 0;
            for (int t = 0; t < deg; ++t) {
                const int v = s[lat.addr(lat.nbr(i, t))];
                eo += (v == old);
                en += (v == nw);
            }
            k = en - eo + D;
        } else if (m.kind == MQV_MODEL_BLUME_CAPEL) {
            // Spin1_Initializer::newsv (src/hamiltonian/util/initializers.h:99-118)
            int st = old;
            if (st == 0) st = rng.real() < 0.5 ? -1 : 1;
            else st = rng.real() < 0.5 ? -st : 0;
            nw = st;
            int sum = 0;
            for (int t = 0; t < deg; ++t) sum += s[lat.addr(lat.nbr(i, t))];
            k = (((nw - old) + 2) * (2 * D + 1) + (sum + D)) * 3 + (nw * nw - old * old + 1);
            if (m.termsel && sub) k += 15 * (2 * D + 1);  // the sublattice-B table
        } else {
            // spin flip (src/hamiltonian/util/initializers.h:52-58), neighbourhood
            // sum with optional bonds (src/libmarqov/metropolishelpers.h:456-537)
            nw = -old;
            int sum = 0;
            for (int t = 0; t < deg; ++t) sum += lat.bond(i, t) * s[lat.addr(lat.nbr(i, t))];
            k = old * sum + D;
        }
        cut = cuts[k];
    }
    // metro_update_accepted (src/libmarqov/metropolis.h:61-64,120-124) on the
    // site's acceptance word, its top byte from the warp's shared table when
    // `tab` is given (accept_tab_fill)
    bool acc;
    if (tab) {
        const uint32_t top = live ? accept_top8_tab(tab, run0, (uint32_t)i) : 0u;
        acc = live && accept_top_or_fine(cut, top, key, (uint32_t)i, sweep, replica);
    } else {
        acc = live && accept_below(cut, key, (uint32_t)i, sweep, replica);
    }
    if (acc) s[ai] = (int8_t)nw;
}

// Site of colour `colour` in pair t of a parity-coloured hypercubic lattice
// with even side: sites 2t and 2t+1 differ only in x, so they have opposite
// colours.
template <class ST>
__device__ __forceinline__ int64_t parity_site(const ST& st, int64_t t, int colour)
{
    const int64_t i0 = 2 * t;
    int par = 0;
    for (int j = 1; j < st.degree(0) / 2; ++j) par += st.coord(i0, j);
    return i0 + (((par & 1) != colour) ? 1 : 0);
}

__device__ __forceinline__ long long warp_sum_ll(long long v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------
// Potts stencils by octets: eight consecutive sites of an x-line as two 32-bit
// words, so a side must be a multiple of 8 and the state row-major.

// 1 in every byte where a and b differ (bytes below 128)
__device__ __forceinline__ uint32_t bytes_differ(uint32_t a, uint32_t b)
{
    return (((a ^ b) + 0x7F7F7F7Fu) >> 7) & 0x01010101u;
}

constexpr int kOctetThreads = kAccSites / 4;

// Call f with the stencil of such a lattice, its dimension fixed.
template <class F>
__device__ __forceinline__ void with_octet_dim(const StencilDev& st, F&& f)
{
    const bool p2 = st.lg >= 0;
    if (st.dim == 2) {
        if (p2) f(StencilDim<2, true>(st));
        else f(StencilDim<2, false>(st));
    } else {
        if (p2) f(StencilDim<3, true>(st));
        else f(StencilDim<3, false>(st));
    }
}

// One aligned block of kAccSites positions of a colour by kOctetThreads threads.
__device__ __forceinline__ void potts_block(const ModelDev& m, const StencilDev& st, int8_t* __restrict__ s, int64_t t0,
                                            int64_t cnt, int colour, Key key, uint32_t sweep, uint32_t replica,
                                            const unsigned long long* __restrict__ cuts, int degree);

// The four sites of colour `colour` in the octet of positions t .. t + 3 (t a
// multiple of 4, all below the colour's count), the same moves as int8_site:
// the sites and each direction's neighbours are four bytes of a word, equal
// neighbours are counted in all four at once, their acceptance bytes come from
// four neighbouring bits of each plane, and the octet is written back whole
// (its other sites are of the other colour: nobody else writes them).
// cuts: the member's table (2 * degree + 1 entries).
// 147 instructions per 32 moves where the per-site kernel takes 302, a third of
// them the draws; a farm of 48 members (2.9 M sites, q = 3): a sweep 40 -> 23 us,
// a measurement 20 -> 5.
template <int D, bool P2>
__device__ __forceinline__ void potts_octet(const ModelDev& m, const StencilDim<D, P2>& st, int8_t* __restrict__ s,
                                            int64_t t, int colour, Key key, uint32_t sweep, uint32_t replica,
                                            const unsigned long long* cuts, const uint4* tab, uint32_t run0)
{
    const uint32_t i0 = 2u * (uint32_t)t, L = (uint32_t)st.len;
    auto load8 = [&](uint32_t i) -> uint2 { return *reinterpret_cast<const uint2*>(s + i); };
    const uint32_t x = (uint32_t)st.coord(i0, 0);
    const uint2 own = load8(i0);
    const uint32_t left = (uint8_t)s[x == 0 ? i0 + L - 1 : i0 - 1], right = (uint8_t)s[x + 8 == L ? i0 + 8 - L : i0 + 8];
    uint2 side[2 * (D - 1)];
    int par = 0;
#pragma unroll
    for (int d = 1; d < D; ++d) {
        const uint32_t p = (uint32_t)st.pow_of(d), w = (L - 1) * p;
        const int c = st.coord(i0, d);
        par += c;
        side[2 * d - 2] = load8(c == (int)L - 1 ? i0 - w : i0 + p);
        side[2 * d - 1] = load8(c == 0 ? i0 + w : i0 - p);
    }
    const uint32_t odd = (uint32_t)((par & 1) != colour);  // the sites' x parity
    const uint32_t sel = odd ? 0x7531u : 0x6420u;
    const uint32_t even4 = __byte_perm(own.x, own.y, 0x6420), odd4 = __byte_perm(own.x, own.y, 0x7531);
    const uint32_t old = odd ? odd4 : even4;
    uint32_t nb[2 * D];
    nb[0] = odd ? (even4 >> 8) | (right << 24) : odd4;
    nb[1] = odd ? even4 : (odd4 << 8) | left;
#pragma unroll
    for (int k = 0; k < 2 * (D - 1); ++k) nb[2 + k] = __byte_perm(side[k].x, side[k].y, sel);
    // proposals (Initializer<Potts<Q>>::newsv): the first word of each site's METRO stream
    uint32_t nw = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        nw |= mod_small(lo64(philox(i0 + odd + 2u * j, sweep, 0u, tag(kMetro, replica), key)), (uint32_t)m.q) << (8 * j);
    // cut index: equal neighbours of the new state less those of the old, plus the degree
    uint32_t k4 = 0x01010101u * (2 * D);
#pragma unroll
    for (int k = 0; k < 2 * D; ++k) k4 += bytes_differ(nb[k], old) - bytes_differ(nb[k], nw);
    // top bytes of the acceptance words: bits q .. q + 3 of the planes, one byte each
    const uint32_t run = (i0 >> 6) - run0, q = (i0 >> 1) & 31u;
    const uint4 pa = tab[(run * 2 + odd) * 2], pb = tab[(run * 2 + odd) * 2 + 1];
    const uint32_t pl[8] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
    uint32_t top4 = 0;
#pragma unroll
    for (int b = 7; b >= 0; --b) top4 = 2u * top4 + ((((pl[b] >> q) & 15u) * 0x00204081u) & 0x01010101u);
    uint32_t res = old;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint64_t cut = cuts[(k4 >> (8 * j)) & 255u];
        if (accept_top_or_fine(cut, (top4 >> (8 * j)) & 255u, key, i0 + odd + 2u * j, sweep, replica))
            res = (res & ~(255u << (8 * j))) | (nw & (255u << (8 * j)));
    }
    const uint32_t e = odd ? even4 : res, o = odd ? res : odd4;
    *reinterpret_cast<uint2*>(s + i0) = make_uint2(__byte_perm(e, o, 0x5140), __byte_perm(e, o, 0x7362));
}

__device__ __forceinline__ void potts_block(const ModelDev& m, const StencilDev& st, int8_t* __restrict__ s, int64_t t0,
                                            int64_t cnt, int colour, Key key, uint32_t sweep, uint32_t replica,
                                            const unsigned long long* __restrict__ cuts, int degree)
{
    __shared__ uint4 tab[kAccTab];
    __shared__ unsigned long long s_cuts[16];
    const uint32_t run0 = (uint32_t)(t0 / 32);
    if (threadIdx.x < 32) accept_tab_fill(tab, run0, key, sweep, replica);
    else if (threadIdx.x - 32 <= 2u * (unsigned)degree) s_cuts[threadIdx.x - 32] = cuts[threadIdx.x - 32];
    __syncthreads();
    const int64_t t = t0 + 4 * threadIdx.x;
    if (t >= cnt) return;
    with_octet_dim(st, [&](const auto& lt) {
        potts_octet(m, lt, s, t, colour, key, sweep, replica, s_cuts, tab, run0);
    });
}

// ---------------------------------------------------------------------------
// measurement: InteractionEnergy / SelfEnergy / Magnetization / PottsMagnetization
// accumulators (src/hamiltonian/util/observables.h:47-65,186-217,251-268,
// src/hamiltonian/Potts.h:46-61), exact in int64.

// Neighbour sum of the interaction energy of site i: sum over nbrs(i) of
// s_i s_j (bonds) or [s_i == s_j] (Potts).  On stencils, where every bond
// appears in both endpoints' lists, twice the sum over the forward
// neighbours (+x, +y, ...) gives the same total with half the loads.
template <class Lat>
__device__ __forceinline__ int int8_bond_sum(const ModelDev& m, const Lat& lat, const int8_t* __restrict__ s,
                                             int64_t i, int si, bool potts)
{
    const int deg = lat.degree(i);
    int loc = 0;
    if (potts)
        for (int t = 0; t < deg; ++t) loc += (s[lat.addr(lat.nbr(i, t))] == si);
    else {
        for (int t = 0; t < deg; ++t) loc += lat.bond(i, t) * s[lat.addr(lat.nbr(i, t))];
        loc *= si;
    }
    return loc;
}
template <class ST, class SP>
__device__ __forceinline__ int int8_bond_sum_stencil(const ST& st, SP s, int64_t i, int si, bool potts)
{
    int loc = 0;
    for (int d = 0; d < st.degree(i) / 2; ++d) {
        const int v = s[st.addr(st.nbr(i, 2 * d))];
        loc += potts ? (v == si) : st.bond(i, 2 * d) * v;
    }
    return 2 * (potts ? loc : loc * si);
}
__device__ __forceinline__ int int8_bond_sum(const ModelDev&, const StencilDev& st, const int8_t* __restrict__ s,
                                             int64_t i, int si, bool potts)
{
    return int8_bond_sum_stencil(st, s, i, si, potts);
}
template <int D, bool P2, bool SPLIT>
__device__ __forceinline__ int int8_bond_sum(const ModelDev&, const StencilDim<D, P2, SPLIT>& st, const int8_t* __restrict__ s,
                                             int64_t i, int si, bool potts)
{
    return int8_bond_sum_stencil(st, s, i, si, potts);
}

// Part `part` of `nparts` of the accumulation (a grid-stride share per CTA;
// the CTA's totals go to acc with atomics).  Potts state counts are
// aggregated per warp (lanes with equal states add once) before the shared
// histogram.
template <class Lat>
__device__ __forceinline__ void measure_int8_part(const ModelDev& m, const Lat& lat, const int8_t* __restrict__ s,
                                                  long long* __restrict__ acc, int64_t part, int64_t nparts)
{
    __shared__ int hist[64];
    __shared__ long long red[3][32];
    const bool potts = m.kind == MQV_MODEL_POTTS;
    if (potts)
        for (int k = threadIdx.x; k < 64; k += blockDim.x) hist[k] = 0;
    __syncthreads();
    long long e = 0, mg = 0, sq = 0;
    const unsigned lane = threadIdx.x & 31;
    // warp-uniform trip count: every lane takes part in the warp's votes
    const int64_t stride = nparts * blockDim.x;
    for (int64_t i0 = part * (int64_t)blockDim.x + (threadIdx.x & ~31u); i0 < lat.n; i0 += stride) {
        const int64_t i = i0 + lane;
        const bool live = i < lat.n;
        int si = 0;
        if (live) {
            si = s[lat.addr(i)];
            e += int8_bond_sum(m, lat, s, i, si, potts);
            mg += si;
            sq += si * si;
        }
        if (potts) {
            const unsigned peers = __match_any_sync(0xffffffffu, live ? (si & 63) : 64);
            if (live && lane == (unsigned)(__ffs(peers) - 1)) atomicAdd(&hist[si & 63], __popc(peers));
        }
    }
    e = warp_sum_ll(e);
    mg = warp_sum_ll(mg);
    sq = warp_sum_ll(sq);
    const int wid = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        red[0][wid] = e;
        red[1][wid] = mg;
        red[2][wid] = sq;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        long long a = 0, b = 0, c = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            a += red[0][k];
            b += red[1][k];
            c += red[2][k];
        }
        atomicAdd(reinterpret_cast<unsigned long long*>(acc + kAccEne), (unsigned long long)a);
        atomicAdd(reinterpret_cast<unsigned long long*>(acc + kAccMag), (unsigned long long)b);
        atomicAdd(reinterpret_cast<unsigned long long*>(acc + kAccSq), (unsigned long long)c);
    }
    if (potts)
        for (int k = threadIdx.x; k < m.q; k += blockDim.x)
            if (hist[k]) atomicAdd(reinterpret_cast<unsigned long long*>(acc + kAccPotts + k), (unsigned long long)hist[k]);
}

// The same of a Potts stencil of at most kOctetStates states by octets: equal
// forward neighbours (each bond lies in both ends' lists: counted twice) and
// the sites of every state, counted in all eight bytes at once.
constexpr int kOctetStates = 8;
template <int D, bool P2>
__device__ __forceinline__ void measure_potts_octets(const ModelDev& m, const StencilDim<D, P2>& st,
                                                     const int8_t* __restrict__ s, long long* __restrict__ acc,
                                                     int64_t part, int64_t nparts)
{
    __shared__ int red[32][kOctetStates + 1];
    const uint32_t L = (uint32_t)st.len, n8 = (uint32_t)(st.n / 8), stride = (uint32_t)(nparts * blockDim.x);
    int bonds = 0, cnt[kOctetStates] = {};
    auto same = [](uint2 a, uint2 b) { return 8 - __popc(bytes_differ(a.x, b.x) | (bytes_differ(a.y, b.y) << 1)); };
    for (uint32_t k = (uint32_t)(part * blockDim.x + threadIdx.x); k < n8; k += stride) {
        const uint32_t i0 = 8u * k, x = (uint32_t)st.coord(i0, 0);
        const uint2 v = *reinterpret_cast<const uint2*>(s + i0);
        const uint32_t right = (uint8_t)s[x + 8 == L ? i0 + 8 - L : i0 + 8];
        uint2 f[D];
        f[0] = make_uint2((v.x >> 8) | (v.y << 24), (v.y >> 8) | (right << 24));
#pragma unroll
        for (int d = 1; d < D; ++d) {
            const uint32_t p = (uint32_t)st.pow_of(d);
            f[d] = *reinterpret_cast<const uint2*>(s + (st.coord(i0, d) == (int)L - 1 ? i0 - (L - 1) * p : i0 + p));
        }
#pragma unroll
        for (int d = 0; d < D; ++d) bonds += same(v, f[d]);
#pragma unroll
        for (int z = 0; z < kOctetStates; ++z)
            if (z < m.q) cnt[z] += same(v, make_uint2(0x01010101u * z, 0x01010101u * z));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bonds = __reduce_add_sync(0xffffffffu, bonds);
    if (lane == 0) red[warp][kOctetStates] = bonds;
#pragma unroll
    for (int z = 0; z < kOctetStates; ++z)
        if (z < m.q) {
            const int c = __reduce_add_sync(0xffffffffu, cnt[z]);
            if (lane == 0) red[warp][z] = c;
        }
    __syncthreads();
    if (threadIdx.x > kOctetStates || (threadIdx.x >= m.q && threadIdx.x < kOctetStates)) return;
    long long sum = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) sum += red[k][threadIdx.x];
    unsigned long long* a = reinterpret_cast<unsigned long long*>(acc);
    const long long z = threadIdx.x;
    if (z == kOctetStates) {
        atomicAdd(a + kAccEne, (unsigned long long)(2 * sum));
    } else if (sum) {
        atomicAdd(a + kAccPotts + z, (unsigned long long)sum);
        if (z) {
            atomicAdd(a + kAccMag, (unsigned long long)(z * sum));
            atomicAdd(a + kAccSq, (unsigned long long)(z * z * sum));
        }
    }
}

// measurement of a stencil
__device__ __forceinline__ void measure_int8_stencil(const ModelDev& m, const StencilDev& st, const int8_t* __restrict__ s,
                                                     long long* __restrict__ acc, int64_t part, int64_t nparts)
{
    if (potts_octets(m, st) && m.q <= kOctetStates) {
        with_octet_dim(st, [&](const auto& lt) { measure_potts_octets(m, lt, s, acc, part, nparts); });
        return;
    }
    with_dim(st, [&](const auto& lt) { measure_int8_part(m, lt, s, acc, part, nparts); });
}

// Accumulators of one measurement -> (e, |m|, m^2, m^4), in the reference's
// order of operations.
__device__ __forceinline__ void finalize_int8_one(const ModelDev& m, int64_t n, const long long* __restrict__ a,
                                                  double* __restrict__ o)
{
    double e, mm;
    if (m.kind == MQV_MODEL_POTTS) {
        long long mx = 0;
        for (int j = 0; j < m.q; ++j) mx = a[kAccPotts + j] > mx ? a[kAccPotts + j] : mx;
        mm = (double)((long long)m.q * mx - n) / (double)(n * (long long)(m.q - 1));
        e = MQV_DMUL(m.k, (double)a[kAccEne]) / (double)(2 * n);
    } else {
        const double mag = (double)a[kAccMag];
        mm = sqrt(MQV_DMUL(mag, mag)) / (double)n;
        e = MQV_DMUL(m.J, (double)a[kAccEne]) / (double)(2 * n);
        // SelfEnergy sums every onsite term over every site, whatever the
        // termselector (observables.h:251-268): (h + h2 terms) / N
        if (m.kind == MQV_MODEL_BLUME_CAPEL)
            e = MQV_DADD(e, MQV_DADD(MQV_DMUL(m.h, (double)a[kAccSq]), MQV_DMUL(m.h2, (double)a[kAccSq])) / (double)n);
    }
    const double m2 = MQV_DMUL(mm, mm);
    o[0] = e;
    o[1] = mm;
    o[2] = m2;
    o[3] = MQV_DMUL(m2, m2);
}

}  // namespace mqv
