// Elementary Monte Carlo steps of small Ising-type lattices (Ising, embedded
// Ising, +-J Edwards-Anderson; 2D and 3D) as bit planes in the shared memory
// of one CTA each, for sm_100a.
//
// The per-site resident kernel (smem_emcs.cu) spends a whole thread on a
// site; a spin is one bit, so here a thread takes a word of 32 sites of an
// x-line through every phase of a chunk of EMCS:
//   * cluster: the candidates are the spin plane or its complement; every bond
//     between two candidates is drawn once from per-warp lists (the draws lie
//     side by side on the lanes); bonds active along x join the sites of a
//     word into runs, a run takes its first neighbour below as its parent by
//     a plain store, the other bonds between runs join the trees by atomic
//     minima; the runs whose root is the seed's are flipped by an exclusive or;
//   * sweep: the acceptance planes of the lattice are drawn once (two Philox
//     blocks per 32 sites), then both colours in turn: anti-aligned neighbours
//     counted by carry-save adders, the tested classes compared with their
//     threshold bytes bit-serially on the 16 active sites of a word; top-byte
//     ties are listed per warp and resolved side by side;
//   * measurement: population counts.
// Same draws, clusters, states and sums as every other path.  Bound by the
// latency of one SM's dependent steps and, in the cluster's bonds, by its
// Philox rate (a block takes a scheduler about 75 cycles per warp).  2D L = 64:
// an EMCS of a cluster, a sweep and a measurement 13.0 us (the per-site kernel
// 24.6), of which the bonds 4.3 and the sweep 2.0.
#include <cuda_runtime.h>

#include <atomic>

#include "batch.h"
#include "resident.h"
#include "runs.cuh"
#include "wolff_int8.cuh"

namespace mqv {

constexpr int kBitsThreads = 512;
constexpr int kBitsWarps = kBitsThreads / 32;
constexpr int kBitsList = 1024;  // bond list entries per warp
constexpr int kBitsRes = kBitsList / 32 + 3;  // outcome words per warp
constexpr int kBitsTies = 64;    // tie list entries per warp
constexpr size_t kBitsHead = kBitsThreads * 4 + 16 + kBitsWarps * 4;  // seed sites, sums, warp totals

// Words of the lattice (every x-line padded to 32 sites) and the layout of
// the shared memory: spins, bond signs, then the sweep's acceptance planes
// and tie lists in the place of the cluster's planes, parents and lists.
struct BitsLayout {
    int wr, nw;         // words per x-line, words
    int edges;          // entries of the cluster's edge list
    size_t runs;        // 64-site runs of the acceptance planes (one past the end)
    size_t spin, sweep, cluster;
    __host__ __device__ BitsLayout(int64_t n, int dim, int len, bool bonds)
    {
        wr = (len + 31) / 32;
        nw = (int)(n / len) * wr;
        runs = (size_t)(n + 63) / 64 + 1;
        spin = ((size_t)nw * 4 * (1 + (bonds ? dim : 0)) + 15) & ~(size_t)15;
        sweep = runs * 64 + (size_t)kBitsWarps * kBitsTies * 16;
        // at most 32 runs a word; edges: 16 a word (more than the densest bond
        // pattern leaves on average; the rest is found again in the planes)
        edges = nw * 16 < kBitsWarps * kBitsList / 2 ? kBitsWarps * kBitsList / 2 : nw * 16;
        const size_t parents = (size_t)nw * 128 > (size_t)kBitsWarps * kBitsRes * 4 ? (size_t)nw * 128 : (size_t)kBitsWarps * kBitsRes * 4;
        cluster = (size_t)nw * 4 * (3 + dim) + parents + (size_t)edges * 4;
    }
    __host__ __device__ size_t bytes(bool clusters) const { return kBitsHead + spin + (clusters && cluster > sweep ? cluster : sweep); }
};
constexpr size_t kBitsMaxSmem = 224 * 1024;

// even bits of x (bits of one parity of a word) packed to 16 bits
__device__ __forceinline__ uint32_t pack16(uint32_t x)
{
    x &= 0x55555555u;
    x = (x | (x >> 1)) & 0x33333333u;
    x = (x | (x >> 2)) & 0x0F0F0F0Fu;
    x = (x | (x >> 4)) & 0x00FF00FFu;
    return (x | (x >> 8)) & 0xFFFFu;
}
__device__ __forceinline__ uint32_t spread16(uint32_t x)
{
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    return (x | (x << 1)) & 0x55555555u;
}

// The lattice's words: neighbours of a word and shifts along its x-line.
template <int D>
struct BitsGeo {
    int L, wr, last;  // side, words per line, sites of a line's last word
    uint64_t mlen;
    int lg;
    __device__ __forceinline__ BitsGeo(const StencilDev& st)
    {
        L = st.len;
        wr = (L + 31) >> 5;
        last = L - 32 * (wr - 1);
        mlen = st.mlen;
        lg = st.lg;
    }
    __device__ __forceinline__ int divL(int r) const
    {
        return lg >= 0 ? r >> lg : (int)__umul64hi((unsigned long long)(uint32_t)r, (unsigned long long)mlen);
    }
    struct Word {
        int wi, row, w, y, z, nb;
    };
    __device__ __forceinline__ Word word(int wi) const
    {
        Word o;
        o.wi = wi;
        o.row = wr == 1 ? wi : wr == 2 ? wi >> 1 : wr == 4 ? wi >> 2 : wi / wr;
        o.w = wi - o.row * wr;
        o.z = D == 3 ? divL(o.row) : 0;
        o.y = o.row - o.z * L;
        o.nb = o.w == wr - 1 ? last : 32;
        return o;
    }
    __device__ __forceinline__ uint32_t valid(const Word& o) const { return 0xFFFFFFFFu >> (32 - o.nb); }
    __device__ __forceinline__ int yp(const Word& o) const { return o.y == L - 1 ? o.wi - (L - 1) * wr : o.wi + wr; }
    __device__ __forceinline__ int ym(const Word& o) const { return o.y == 0 ? o.wi + (L - 1) * wr : o.wi - wr; }
    __device__ __forceinline__ int zp(const Word& o) const { return o.z == L - 1 ? o.wi - (L - 1) * L * wr : o.wi + L * wr; }
    __device__ __forceinline__ int zm(const Word& o) const { return o.z == 0 ? o.wi + (L - 1) * L * wr : o.wi - L * wr; }
    __device__ __forceinline__ int xpw(const Word& o) const { return o.w == wr - 1 ? o.wi - (wr - 1) : o.wi + 1; }
    __device__ __forceinline__ int xmw(const Word& o) const { return o.w == 0 ? o.wi + (wr - 1) : o.wi - 1; }
    // the plane's bits at x + 1 and x - 1 of every site of the word
    __device__ __forceinline__ uint32_t xp(const uint32_t* a, const Word& o, uint32_t v) const
    {
        return (v >> 1) | ((a[xpw(o)] & 1u) << (o.nb - 1));
    }
    __device__ __forceinline__ uint32_t xm(const uint32_t* a, const Word& o, uint32_t v) const
    {
        return (v << 1) | ((a[xmw(o)] >> (o.w == 0 ? last - 1 : 31)) & 1u);
    }
};

// the tested classes of a sweep: q anti-aligned neighbours, u53 threshold T
// below 2^53 (at most half the degree of them), as lane masks
struct BitsClasses {
    unsigned long long T[3];
    uint32_t c0[3], c1[3], c2[3];  // bits of q, inverted: mask = ~((q0 ^ ..) | ..)
    uint32_t t8[3];
    uint32_t zt[3];
    int count;
};

template <int D, bool BOND>
__device__ void bits_run(const ResidentRun& R, unsigned char* smem)
{
    int* s_rsite = reinterpret_cast<int*>(smem);  // seed sites drawn ahead
    int* s_sum = s_rsite + kBitsThreads;
    int &s_size = s_sum[2], &s_nedge = s_sum[3];
    int* s_warp = s_sum + 4;
    smem += kBitsHead;
    const int64_t n = R.st.n;
    const BitsLayout lay(n, D, R.st.len, BOND);
    const BitsGeo<D> g(R.st);
    const int NW = lay.nw, L = g.L;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t* A = reinterpret_cast<uint32_t*>(smem);  // spins, set: -1
    uint32_t* NB = A + NW;                            // +d bonds, set: -1 (plane d at NB + d NW)
    // sweep
    uint4* tab = reinterpret_cast<uint4*>(smem + lay.spin);
    uint4* ties = tab + lay.runs * 4 + warp * kBitsTies;
    // cluster
    uint32_t* sC = reinterpret_cast<uint32_t*>(smem + lay.spin);
    uint32_t* sS = sC + NW;
    uint32_t* sB = sS + NW;  // active bonds, plane d at sB + d NW
    int* sR = reinterpret_cast<int*>(sB + D * NW);  // first run of every word
    int* P = sR + NW;                                // parents of the runs
    // the warps' bond lists, then the edges between runs
    uint32_t* edge = reinterpret_cast<uint32_t*>(P + (NW * 32 > kBitsWarps * kBitsRes ? NW * 32 : kBitsWarps * kBitsRes));
    unsigned short* list = reinterpret_cast<unsigned short*>(edge) + warp * kBitsList;
    uint32_t* res = reinterpret_cast<uint32_t*>(P) + warp * kBitsRes;  // outcomes of the list (before there are runs)

    // The state (and the bond signs) to planes: a thread takes 64 sites of split
    // rows, or a word of a line of a multiple of 8 sites, in wide loads; else the
    // warps take word by word, several words' loads in flight.
    // (A call of one EMCS is mostly this: 32 members of L = 128, a sweep and an
    // exchange per launch 29.6 -> 16.4 us, of L = 160 51 -> 20.)
    const bool split = R.st.split, wide = split || L % 8 == 0;
    if (!BOND && split) {
        for (int k = tid; k < NW / 2; k += kBitsThreads) {
            const int row = g.wr == 2 ? k : 2 * k / g.wr, h = k - row * (g.wr / 2);
            const uint4* q = reinterpret_cast<const uint4*>(R.state + (int64_t)row * L + 32 * h);
            const uint4* q1 = reinterpret_cast<const uint4*>(R.state + (int64_t)row * L + L / 2 + 32 * h);
            const uint4 e0 = q[0], e1 = q[1], o0 = q1[0], o1 = q1[1];
            const uint32_t E = pack_word(e0, e1), O = pack_word(o0, o1);
            A[2 * k] = spread16(E & 0xFFFFu) | (spread16(O & 0xFFFFu) << 1);
            A[2 * k + 1] = spread16(E >> 16) | (spread16(O >> 16) << 1);
        }
    } else if (wide) {
        // plane 0: the spins, plane 1 + d: the +d bonds
        for (int k = tid; k < (BOND ? 1 + D : 1) * NW; k += kBitsThreads) {
            const int d = BOND ? k / NW : 0, wi = k - d * NW;
            const auto o = g.word(wi);
            const int8_t* p = (d == 0 ? R.state : R.st.fb + (int64_t)(d - 1) * n) + (int64_t)o.row * L + 32 * o.w;
            uint2 v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = 8 * j < o.nb ? reinterpret_cast<const uint2*>(p)[j] : make_uint2(0u, 0u);
            uint32_t m = 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) m |= (pack4(v[j].x) | (pack4(v[j].y) << 4)) << (8 * j);
            A[k] = m;  // the bonds' planes follow the spins'
        }
    } else {
        constexpr int NLD = BOND ? 4 : 8;
        for (int w0 = warp; w0 < NW; w0 += NLD * kBitsWarps) {
            int8_t v[NLD][BOND ? 1 + D : 1];
#pragma unroll
            for (int k = 0; k < NLD; ++k) {
                const int wi = w0 + k * kBitsWarps;
                const auto o = g.word(wi < NW ? wi : 0);
                const int x = 32 * o.w + lane;
                const bool live = wi < NW && x < L;
                const int64_t i = live ? (int64_t)o.row * L + x : 0;
                v[k][0] = live ? R.state[R.st.addr(i)] : (int8_t)0;
                if (BOND)
#pragma unroll
                    for (int d = 0; d < D; ++d) v[k][1 + d] = live ? R.st.fb[(int64_t)d * n + i] : (int8_t)0;
            }
#pragma unroll
            for (int k = 0; k < NLD; ++k) {
                const int wi = w0 + k * kBitsWarps;
#pragma unroll
                for (int d = 0; d < (BOND ? 1 + D : 1); ++d) {
                    const uint32_t m = __ballot_sync(0xffffffffu, v[k][d] < 0);
                    if (lane == 0 && wi < NW) A[d * NW + wi] = m;  // the bonds' planes follow the spins'
                }
            }
        }
    }
    if (tid < 2) s_sum[tid] = 0;
    BitsClasses cl;
    cl.count = 0;
#pragma unroll
    for (int c = 0; c < D; ++c) {
        cl.T[c] = 0;
        cl.t8[c] = 0;
        cl.zt[c] = 0;
        cl.c0[c] = cl.c1[c] = cl.c2[c] = 0;
    }
    if (R.nmetro > 0) {
#pragma unroll
        for (int q = 0; q <= 2 * D; ++q) {
            const unsigned long long T = R.cuts[2 * (2 * D - q)];
            if (T >= (1ull << 53)) continue;
#pragma unroll
            for (int c = 0; c < D; ++c)
                if (c == cl.count) {
                    cl.T[c] = T;
                    cl.t8[c] = (uint32_t)(T >> 45);
                    cl.zt[c] = (T & ((1ull << 45) - 1)) == 0 ? 0u : 0xFFFFFFFFu;
                    cl.c0[c] = 0u - (uint32_t)(q & 1);
                    cl.c1[c] = 0u - (uint32_t)((q >> 1) & 1);
                    cl.c2[c] = 0u - (uint32_t)((q >> 2) & 1);
                }
            ++cl.count;
        }
    }
    __syncthreads();

    const uint32_t tgs = tag(kWolffSeed, R.replica), tgb = tag(kWolffBond, R.replica);
    const uint32_t c3a = tag(kAccept, R.replica);
    // lanes per word in the cluster's phases: as many as keep every warp busy
    const int lw = NW * 8 <= kBitsThreads ? 3 : NW * 4 <= kBitsThreads ? 2 : NW * 2 <= kBitsThreads ? 1 : 0;
    const int LPW = 1 << lw, per = 32 >> lw, chunk = kBitsThreads >> lw;
    const uint32_t part = (lw == 0 ? 0xFFFFFFFFu : (1u << per) - 1u) << (per * (lane & (LPW - 1)));
    int nseed = 0;  // seeds drawn ahead, s_rsite[0 .. kBitsThreads)
    for (int e = 0; e < R.n_emcs; ++e) {
        for (int c = 0; c < R.ncluster; ++c) {
            const int k = e * R.ncluster + c;
            const uint32_t serial = R.cluster0 + (uint32_t)k;
            if (k >= nseed) {
                // the next seed sites, one per thread (wolff_int8_seed's first word)
                __syncthreads();
                s_rsite[tid] = (int)(lo64(philox(0u, serial + (uint32_t)tid, 0u, tgs, R.key)) % (uint64_t)n);
                nseed = k + kBitsThreads;
                __syncthreads();
            }
            const uint32_t rsite = (uint32_t)s_rsite[k - (nseed - kBitsThreads)];
            const int srow = g.divL((int)rsite), sx = (int)rsite - srow * L, sw = srow * g.wr + (sx >> 5);
            const uint32_t flip = ((A[sw] >> (sx & 31)) & 1u) ? 0u : 0xFFFFFFFFu;  // candidates: A ^ flip
            if (tid == 0) s_size = 0;
            for (int wi = tid; wi < NW; wi += kBitsThreads) {
                const auto o = g.word(wi);
                sC[wi] = (A[wi] ^ flip) & g.valid(o);
            }
            __syncthreads();
            // Active bonds: the bonds between two candidates are listed per warp,
            // all directions in one list where it holds them, and drawn side by
            // side over the lanes; the outcomes come back as a bit string in
            // the list's order.
            const WolffDev w = R.w;
            const RoundKeys key(R.key);
            const int dstep = per * 32 * D <= kBitsList ? D : 1;
            for (int w0 = 0; w0 < NW; w0 += chunk) {
                const int wb = w0 + warp * per;  // the warp's first word
                const int wi = wb + (lane >> lw);
                const bool inw = wi < NW;
                const auto o = g.word(inw ? wi : 0);
                const uint32_t C = inw ? sC[wi] & part : 0u;
                const uint32_t base = (uint32_t)(o.row * L + 32 * o.w);
                const uint32_t endx = o.w == g.wr - 1 ? (uint32_t)(o.nb - 1) : 32u;  // bit of the line's last site
                const uint32_t offy = o.y == L - 1 ? (uint32_t)(L - L * L) : (uint32_t)L;
                const uint32_t offz = D == 3 ? (o.z == L - 1 ? (uint32_t)(L * L - L * L * L) : (uint32_t)(L * L)) : 0u;
                for (int d0 = 0; d0 < D; d0 += dstep) {
                    uint32_t Q[D];
                    int cnt = 0;
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        Q[d] = 0u;
                        if (d >= d0 && d < d0 + dstep && inw)
                            Q[d] = C & (d == 0 ? g.xp(sC, o, sC[wi]) : sC[d == 1 ? g.yp(o) : g.zp(o)]);
                        cnt += __popc(Q[d]);
                    }
                    int pos = warp_prefix(cnt, lane);
                    const int total = __shfl_sync(0xffffffffu, pos, 31);
                    const int first = pos -= cnt;
                    __syncwarp();
#pragma unroll
                    for (int d = 0; d < D; ++d)
                        for (uint32_t m = Q[d]; m; m &= m - 1)
                            list[pos++] = (unsigned short)((d << 10) | ((lane >> lw) << 5) | (__ffs(m) - 1));
                    __syncwarp();
                    for (int k0 = 0; k0 < total; k0 += 64) {
                        // two bonds side by side; a word's first site and the
                        // way to its neighbours come from the lane that holds it
                        uint32_t lo[2], hi[2];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int q = k0 + 32 * h + lane;
                            const uint32_t id = list[q < total ? q : 0], b = id & 31u;
                            const int src = (int)((id >> 5) & 31u) << lw, d = (int)(id >> 10);
                            const uint32_t i = __shfl_sync(0xffffffffu, base, src) + b;
                            const uint32_t oy = __shfl_sync(0xffffffffu, offy, src);
                            const uint32_t ox = __shfl_sync(0xffffffffu, endx, src) == b ? 1u - (uint32_t)L : 1u;
                            uint32_t off = d == 0 ? ox : oy;
                            if (D == 3) {
                                const uint32_t oz = __shfl_sync(0xffffffffu, offz, src);
                                off = d == 2 ? oz : off;
                            }
                            const uint32_t j = i + off;
                            lo[h] = min(i, j);
                            hi[h] = max(i, j);
                        }
                        const bool a0 = wolff_int8_active(w, lo[0], hi[0], serial, tgb, key);
                        const bool a1 = wolff_int8_active(w, lo[1], hi[1], serial, tgb, key);
                        const uint32_t r0 = __ballot_sync(0xffffffffu, a0), r1 = __ballot_sync(0xffffffffu, a1);
                        if (lane == 0) {
                            res[k0 >> 5] = r0;
                            res[(k0 >> 5) + 1] = r1;
                        }
                    }
                    __syncwarp();
                    uint32_t bits = bit_string(res, first);  // at most 32 bonds a lane
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        if (d < d0 || d >= d0 + dstep) continue;
                        const int nb = __popc(Q[d]);
                        const uint32_t B = group_or(bit_deposit(bits, Q[d]), LPW);
                        bits = nb < 32 ? bits >> nb : 0u;
                        if (inw && (lane & (LPW - 1)) == 0) sB[d * NW + wi] = B;
                    }
                }
            }
            __syncthreads();
            // Runs: the bonds along x join the sites of a word.  They are
            // numbered through (sR: first run of every word), so that the
            // steps below take one run or edge per thread without loops over
            // the bits of a word.
            if (tid == 0) s_nedge = 0;
            int nrun = 0;  // runs of the words before the round's
            for (int w0 = 0; w0 < NW; w0 += kBitsThreads) {
                const int wi = w0 + tid;
                uint32_t S = 0u;
                if (wi < NW) {
                    S = sC[wi] & ~((sB[wi] & (g.valid(g.word(wi)) >> 1)) << 1);
                    sS[wi] = S;
                }
                const int cnt = __popc(S);
                const int pos = warp_prefix(cnt, lane);
                if (lane == 31) s_warp[warp] = pos;
                __syncthreads();
                int before = warp_prefix(lane < kBitsWarps ? s_warp[lane] : 0, lane);
                const int total = __shfl_sync(0xffffffffu, before, kBitsWarps - 1);
                before = __shfl_sync(0xffffffffu, before, warp) - s_warp[warp];
                if (wi < NW) sR[wi] = nrun + before + pos - cnt;
                nrun += total;
                __syncthreads();
            }
            for (int k2 = tid; k2 < nrun; k2 += kBitsThreads) P[k2] = k2;
            __syncthreads();
            // the run of bit b of word wj
            auto run_of = [&](int wj, int b) { return sR[wj] + __popc(sS[wj] & (0xFFFFFFFFu >> (31 - b))) - 1; };
            // A run's first neighbour below (no periodic bond) becomes its parent
            // by a plain store; the further bonds between runs, one per pair
            // where they are adjacent, are the edges left, listed.
            const int cap = lay.edges;
            for (int w0 = 0; w0 < NW; w0 += chunk) {
                const int wi = w0 + (tid >> lw);
                const bool inw = wi < NW;
                const auto o = g.word(inw ? wi : 0);
                const int wm = g.ym(o), wz = D == 3 ? g.zp(o) : 0;
                uint32_t ey = 0u, ez = 0u, ex = 0u;
                if (inw) {
                    const uint32_t X = sB[wi] & (g.valid(o) >> 1), Y = sB[NW + wm];
                    ey = Y & ~((Y & X & sB[wm]) << 1) & part;
                    if (o.y != 0) {
                        const uint32_t above = run_above(Y, X);
                        for (uint32_t m = Y & ~above & part; m; m &= m - 1) {
                            const int b = __ffs(m) - 1;
                            P[run_of(wi, b)] = run_of(wm, b);
                        }
                        ey &= above;
                    }
                    if (D == 3) {
                        const uint32_t Z = sB[2 * NW + wi];
                        ez = Z & ~((Z & X & sB[wz]) << 1) & part;
                    }
                    ex = sB[wi] & (1u << (o.nb - 1)) & part;  // from the word's last site to the next word
                }
                const int cnt = __popc(ey) + __popc(ez) + (ex ? 1 : 0);
                const int pos = warp_prefix(cnt, lane);
                int at = 0;
                if (lane == 31 && pos) at = atomicAdd(&s_nedge, pos);
                at = __shfl_sync(0xffffffffu, at, 31) + pos - cnt;
                auto put = [&](uint32_t m, int wj, bool next) {
                    for (; m; m &= m - 1) {
                        const int b = __ffs(m) - 1;
                        if (at < cap) edge[at] = (uint32_t)run_of(wi, b) | ((uint32_t)run_of(wj, next ? 0 : b) << 16);
                        ++at;
                    }
                };
                put(ey, wm, false);
                if (D == 3) put(ez, wz, false);
                put(ex, inw ? g.xpw(o) : 0, true);
            }
            __syncthreads();
            const int nedge = s_nedge < cap ? s_nedge : cap;
            const bool over = s_nedge > cap;  // the edges that the list does not hold are found in the planes again
            forest_jump(P, nrun, tid, kBitsThreads);
            __syncthreads();
            for (int k2 = tid; k2 < nedge; k2 += kBitsThreads) {
                const uint32_t e2 = edge[k2];
                forest_join(P, (int)(e2 & 0xFFFFu), (int)(e2 >> 16));
            }
            if (over)
                for (int wi = tid; wi < NW; wi += kBitsThreads) {
                    const auto o = g.word(wi);
                    for (uint32_t m = sB[NW + wi]; m; m &= m - 1)
                        forest_join(P, run_of(wi, __ffs(m) - 1), run_of(g.yp(o), __ffs(m) - 1));
                    if (D == 3)
                        for (uint32_t m = sB[2 * NW + wi]; m; m &= m - 1)
                            forest_join(P, run_of(wi, __ffs(m) - 1), run_of(g.zp(o), __ffs(m) - 1));
                    if (sB[wi] & (1u << (o.nb - 1))) forest_join(P, run_of(wi, o.nb - 1), run_of(g.xpw(o), 0));
                }
            __syncthreads();
            forest_jump(P, nrun, tid, kBitsThreads);
            __syncthreads();
            // flip the runs below the seed's root: a bit per run, in order
            {
                const int root = P[run_of(sw, sx & 31)];
                uint32_t* hit = edge;
                for (int k0 = warp * 32; k0 < nrun + 32; k0 += kBitsThreads) {
                    const int k2 = k0 + lane;
                    const uint32_t m = __ballot_sync(0xffffffffu, k2 < nrun && P[k2] == root);
                    if (lane == 0) hit[k0 >> 5] = m;
                }
                __syncthreads();
                int size = 0;
                for (int w0 = 0; w0 < NW; w0 += chunk) {
                    const int wi = w0 + (tid >> lw);
                    const bool inw = wi < NW;
                    const uint32_t S = inw ? sS[wi] : 0u, mine = S & part;
                    const int k2 = inw ? sR[wi] + __popc(S & (part - 1u) & ~part) : 0;
                    uint32_t f = mine ? bit_deposit(bit_string(hit, k2), mine) : 0u;
                    f = group_or(f, LPW);
                    if (inw && (lane & (LPW - 1)) == 0 && f) {
                        f = run_fill(f, sB[wi] & (g.valid(g.word(wi)) >> 1));
                        A[wi] ^= f;
                        size += __popc(f);
                    }
                }
                size = __reduce_add_sync(0xffffffffu, size);
                if (lane == 0 && size) atomicAdd(&s_size, size);
            }
            __syncthreads();
            if (tid == 0) R.csize[e * R.csize_e + c * R.csize_c] = s_size;
        }
        for (int j = 0; j < R.nmetro; ++j) {
            const uint32_t sweep = R.sweep0 + (uint32_t)(e * R.nmetro + j);
            // the lattice's acceptance planes: run, parity, half
            for (int k = tid; k < (int)(lay.runs - 1) * 4; k += kBitsThreads)
                tab[k] = philox(((uint32_t)k >> 2) * 2u + (((uint32_t)k >> 1) & 1u), sweep, (uint32_t)k & 1u, c3a, R.key);
            __syncthreads();
            for (int colour = 0; colour < 2; ++colour) {
                int ntie = 0;
                auto flush = [&]() {
                    __syncwarp();
                    for (int q = lane; q < ntie; q += 32) {
                        const uint4 te = ties[q];
                        const auto o = g.word((int)(te.x >> 1));
                        const uint32_t p = te.x & 1u, i0 = (uint32_t)(o.row * L + 32 * o.w);
                        uint32_t flips = 0u;
                        for (uint32_t m = te.y; m; m &= m - 1) {
                            const int b = __ffs(m) - 1;
                            const int c = ((te.z >> b) & 1u) ? 0 : ((te.w >> b) & 1u) ? 1 : 2;
                            unsigned long long T = cl.T[0];
                            uint32_t t8 = cl.t8[0];
#pragma unroll
                            for (int v = 1; v < D; ++v)
                                if (c == v) {
                                    T = cl.T[v];
                                    t8 = cl.t8[v];
                                }
                            const uint64_t fine = accept_fine56(R.key, i0 + 2u * (uint32_t)b + p, sweep, R.replica);
                            if ((((uint64_t)t8 << 45) | (fine >> 11)) < T) flips |= 1u << (2 * b + (int)p);
                        }
                        if (flips) atomicXor(&A[o.wi], flips);
                    }
                    __syncwarp();
                    ntie = 0;
                };
                for (int w0 = warp * 32; w0 < NW; w0 += kBitsThreads) {
                    const int wi = w0 + lane;
                    uint32_t tie = 0u, mA = 0u, mB = 0u, ent = 0u;
                    if (wi < NW) {
                        const auto o = g.word(wi);
                        const uint32_t p = (uint32_t)(colour + o.y + o.z) & 1u;
                        const uint32_t a = A[wi];
                        // anti-aligned neighbours, one bit plane each
                        uint32_t v[2 * D];
                        v[0] = a ^ g.xp(A, o, a);
                        v[1] = a ^ g.xm(A, o, a);
                        v[2] = a ^ A[g.yp(o)];
                        v[3] = a ^ A[g.ym(o)];
                        if (D == 3) {
                            v[2 * D - 2] = a ^ A[g.zp(o)];
                            v[2 * D - 1] = a ^ A[g.zm(o)];
                        }
                        if (BOND) {
                            const uint32_t bx = NB[wi];
                            v[0] ^= bx;
                            v[1] ^= g.xm(NB, o, bx);
                            v[2] ^= NB[NW + wi];
                            v[3] ^= NB[NW + g.ym(o)];
                            if (D == 3) {
                                v[2 * D - 2] ^= NB[2 * NW + wi];
                                v[2 * D - 1] ^= NB[2 * NW + g.zm(o)];
                            }
                        }
                        // their number q (carry-save adders)
                        const uint32_t s3 = v[0] ^ v[1] ^ v[2], k3 = (v[0] & v[1]) | (v[2] & (v[0] | v[1]));
                        uint32_t q0, q1, q2;
                        if (D == 2) {
                            const uint32_t k4 = s3 & v[3];
                            q0 = s3 ^ v[3];
                            q1 = k3 ^ k4;
                            q2 = k3 & k4;
                        } else {
                            const uint32_t s6 = v[3] ^ v[2 * D - 2] ^ v[2 * D - 1],
                                           k6 = (v[3] & v[2 * D - 2]) | (v[2 * D - 1] & (v[3] | v[2 * D - 2]));
                            const uint32_t k0 = s3 & s6;
                            q0 = s3 ^ s6;
                            q1 = k3 ^ k6 ^ k0;
                            q2 = (k3 & k6) | (k0 & (k3 | k6));
                        }
                        // the tested classes on the 16 active sites
                        const uint32_t act = (p ? 0xAAAAAAAAu : 0x55555555u) & g.valid(o);
                        uint32_t m[D];
                        uint32_t test = 0u;
#pragma unroll
                        for (int c = 0; c < D; ++c) {
                            m[c] = 0u;
                            if (c < cl.count) {
                                m[c] = ~((q0 ^ cl.c0[c]) | (q1 ^ cl.c1[c]) | (q2 ^ cl.c2[c])) & act;
                                m[c] = pack16(m[c] >> p);
                                test |= m[c];
                            }
                        }
                        const uint32_t i0 = (uint32_t)(o.row * L + 32 * o.w), sh = (i0 >> 1) & 31u;
                        const uint4* t = tab + (((i0 >> 6) << 1) + p) * 2;
                        const uint4 lo0 = t[0], lo1 = t[1];
                        uint4 hi0 = lo0, hi1 = lo1;
                        if (sh > 16u) {  // the word's sites straddle two runs
                            hi0 = t[4];
                            hi1 = t[5];
                        }
                        const uint32_t lo[8] = {lo0.x, lo0.y, lo0.z, lo0.w, lo1.x, lo1.y, lo1.z, lo1.w};
                        const uint32_t hi[8] = {hi0.x, hi0.y, hi0.z, hi0.w, hi1.x, hi1.y, hi1.z, hi1.w};
                        uint32_t borrow = 0u, eq = ~0u;
#pragma unroll
                        for (int b = 0; b < 8; ++b) {
                            uint32_t tb = 0u;
#pragma unroll
                            for (int c = 0; c < D; ++c) tb |= m[c] & (0u - ((cl.t8[c] >> b) & 1u));
                            const uint32_t x = __funnelshift_r(lo[b], hi[b], sh), nx = ~x;
                            borrow = (nx & (tb | borrow)) | (tb & borrow);
                            eq &= ~(x ^ tb);
                        }
                        uint32_t open = 0u;  // classes whose tie needs the fine block
#pragma unroll
                        for (int c = 0; c < D; ++c) open |= m[c] & cl.zt[c];
                        tie = eq & open;
                        mA = m[0];
                        mB = m[1];
                        ent = ((uint32_t)wi << 1) | p;
                        // accepted: the sites outside the tested classes and those below their threshold
                        const uint32_t no = spread16(test & ~borrow) << p;
                        A[wi] = a ^ (act & ~no);
                    }
                    const uint32_t has = __ballot_sync(0xffffffffu, tie != 0u);
                    if (has) {
                        if (ntie + __popc(has) > kBitsTies) flush();
                        if (tie) ties[ntie + __popc(has & ((1u << lane) - 1u))] = make_uint4(ent, tie, mA, mB);
                        ntie += __popc(has);
                    }
                }
                if (ntie) flush();
                __syncthreads();
            }
        }
        if (R.acc) {
            if (R.ncluster == 0 && R.nmetro == 0) __syncthreads();  // the sums were set to zero by thread 0
            int anti = 0, minus = 0;
            for (int wi = tid; wi < NW; wi += kBitsThreads) {
                const auto o = g.word(wi);
                const uint32_t a = A[wi], vm = g.valid(o);
                uint32_t vx = a ^ g.xp(A, o, a), vy = a ^ A[g.yp(o)], vz = D == 3 ? a ^ A[g.zp(o)] : 0u;
                if (BOND) {
                    vx ^= NB[wi];
                    vy ^= NB[NW + wi];
                    if (D == 3) vz ^= NB[2 * NW + wi];
                }
                anti += __popc(vx & vm) + __popc(vy & vm) + (D == 3 ? __popc(vz & vm) : 0);
                minus += __popc(a);
            }
            anti = __reduce_add_sync(0xffffffffu, anti);
            minus = __reduce_add_sync(0xffffffffu, minus);
            if (lane == 0) {
                atomicAdd(&s_sum[0], anti);
                atomicAdd(&s_sum[1], minus);
            }
            __syncthreads();
            if (tid == 0) {
                // sum_i s_i sum_{j in nbrs(i)} s_j counts every bond twice
                long long* acc = R.acc + e * R.acc_e;
                acc[kAccEne] = 2ll * ((long long)D * n - 2ll * s_sum[0]);
                acc[kAccMag] = n - 2ll * s_sum[1];
                acc[kAccSq] = n;
                s_sum[0] = s_sum[1] = 0;
            }
        }
    }
    __syncthreads();
    if (!BOND && split) {
        for (int k = tid; k < NW / 2; k += kBitsThreads) {
            const int row = g.wr == 2 ? k : 2 * k / g.wr, h = k - row * (g.wr / 2);
            const uint32_t a = A[2 * k], b = A[2 * k + 1];
            uint4 lo, hi;
            uint4* q = reinterpret_cast<uint4*>(R.state + (int64_t)row * L + 32 * h);
            unpack_word(pack16(a) | (pack16(b) << 16), lo, hi);
            q[0] = lo;
            q[1] = hi;
            q = reinterpret_cast<uint4*>(R.state + (int64_t)row * L + L / 2 + 32 * h);
            unpack_word(pack16(a >> 1) | (pack16(b >> 1) << 16), lo, hi);
            q[0] = lo;
            q[1] = hi;
        }
    } else if (wide) {
        for (int wi = tid; wi < NW; wi += kBitsThreads) {
            const auto o = g.word(wi);
            const uint32_t a = A[wi];
            uint2* p = reinterpret_cast<uint2*>(R.state + (int64_t)o.row * L + 32 * o.w);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (8 * j < o.nb) p[j] = make_uint2(unpack4((a >> (8 * j)) & 15u), unpack4((a >> (8 * j + 4)) & 15u));
        }
    } else {
        for (int wi = warp; wi < NW; wi += kBitsWarps) {
            const auto o = g.word(wi);
            const int x = 32 * o.w + lane;
            if (x < L) R.state[R.st.addr((int64_t)o.row * L + x)] = (A[wi] >> lane) & 1u ? -1 : 1;
        }
    }
}

template <int D, bool BOND>
__global__ void __launch_bounds__(kBitsThreads, 1) bits_emcs(ResidentRun R)
{
    extern __shared__ __align__(16) unsigned char smem[];
    bits_run<D, BOND>(R, smem);
}

// One CTA per member of `order` (the batch's bit-plane members, largest
// first): EMCS e0 .. e0 + count - 1 of the run, measurement slots slot0 ..
__global__ void __launch_bounds__(kBitsThreads, 1)
    batch_bits(const BatchRep* __restrict__ reps, const int32_t* __restrict__ order, int nrep, uint32_t e0, int slot0,
               int count, int ncluster, int nmetro, long long* __restrict__ acc, int32_t* __restrict__ csize)
{
    extern __shared__ __align__(16) unsigned char smem[];
    grid_dep_launch();
    grid_dep_wait();
    const int r = order[blockIdx.x];
    ResidentRun R;
    resident_member(R, reps[r], r, nrep, e0, slot0, count, ncluster, nmetro, acc, csize);
    if (R.st.fb) {
        if (R.st.dim == 2) bits_run<2, true>(R, smem);
        else bits_run<3, true>(R, smem);
    } else {
        if (R.st.dim == 2) bits_run<2, false>(R, smem);
        else bits_run<3, false>(R, smem);
    }
}

bool bits_fits(const Sim* s, bool clusters)
{
    if (s->is_f32 || s->lat_kind != MQV_LATTICE_HYPERCUBIC || s->dim < 2 || s->dim > 3) return false;
    if (s->md.kind != MQV_MODEL_ISING && s->md.kind != MQV_MODEL_ISING_EMBED && s->md.kind != MQV_MODEL_EA) return false;
    if (s->d_bonds && !s->bonds_unit) return false;
    if (s->n > (1 << 20)) return false;
    return BitsLayout(s->n, s->dim, s->len, s->d_bonds != nullptr).bytes(clusters) <= kBitsMaxSmem;
}
size_t bits_smem(const Sim* s, bool clusters)
{
    return BitsLayout(s->n, s->dim, s->len, s->d_bonds != nullptr).bytes(clusters);
}

static cudaError_t bits_attr(int device)
{
    static std::atomic<bool> done[64] = {};  // host threads share it
    if (device >= 0 && device < 64 && done[device]) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    const void* k[5] = {(const void*)bits_emcs<2, false>, (const void*)bits_emcs<2, true>, (const void*)bits_emcs<3, false>,
                        (const void*)bits_emcs<3, true>, (const void*)batch_bits};
    for (const void* f : k)
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBitsMaxSmem);
    if (e == cudaSuccess && device >= 0 && device < 64) done[device] = true;
    return e;
}

cudaError_t launch_bits_emcs(const ResidentRun& R, bool bonds, cudaStream_t st, int device)
{
    const cudaError_t e = bits_attr(device);
    if (e != cudaSuccess) return e;
    const size_t smem = BitsLayout(R.st.n, R.st.dim, R.st.len, bonds).bytes(R.ncluster > 0);
    if (R.st.dim == 2) {
        if (bonds) bits_emcs<2, true><<<1, kBitsThreads, smem, st>>>(R);
        else bits_emcs<2, false><<<1, kBitsThreads, smem, st>>>(R);
    } else {
        if (bonds) bits_emcs<3, true><<<1, kBitsThreads, smem, st>>>(R);
        else bits_emcs<3, false><<<1, kBitsThreads, smem, st>>>(R);
    }
    return cudaGetLastError();
}

cudaError_t batch_launch_bits(const BatchLaunch& b, cudaStream_t st, const int32_t* order, int nmem, size_t smem,
                              uint32_t e0, int slot0, int count, int ncluster, int nmetro, int device)
{
    if (nmem <= 0 || count <= 0) return cudaSuccess;
    const cudaError_t e = bits_attr(device);
    if (e != cudaSuccess) return e;
    return launch_pdl_smem(batch_bits, (unsigned)nmem, kBitsThreads, smem, st, b.reps, order, b.nrep, e0, slot0, count,
                           ncluster, nmetro, b.acc, b.csize);
}

}  // namespace mqv
