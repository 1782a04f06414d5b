// Fused checkerboard Metropolis sweep for the 2D Ising model on sm_100a,
// bit-sliced in shared memory.
//
// HBM layout ("split rows"): row y of the L x L lattice is stored as its L/2
// even-x sites followed by its L/2 odd-x sites, int8 +-1.  Sites of one colour
// in a row are then contiguous, and the neighbours of element j of one half
// are element j of the same half in the rows above and below and elements
// j-1, j (even half) or j, j+1 (odd half) of the other half of the row.
//
// Pipeline: every warp is an independent worker with its own shared-memory
// partition.  It takes TY x TX tiles from a global tile counter; the rows of a
// tile plus a two-row / 64-column halo of the old state stream in through an
// 8-row staging ring filled by the bulk-copy engine (cp.async.bulk, one
// mbarrier per slot), are packed to bits as they arrive, and the updated rows
// leave through an output ring drained by bulk stores to the other state
// buffer.  Loads for the next tile are in flight while the warp updates the
// current one; the warp only ever synchronises with itself.  Every site is
// read from HBM once and written once per sweep (2 bytes).  Tile shape and
// warps per CTA are picked per lattice size by timing the candidates.
//
// Each staged half-row is packed to one bit per site (1 = spin -1) in 32-site
// words.  Colour 0 is updated on the tile and its
// one-site ring (re-deriving the neighbouring tiles' updates, which are
// deterministic), then colour 1 on the tile; a 32-site word costs a few dozen
// logic instructions: neighbour counts by a carry-save adder on the bit
// planes, the site class (number of aligned neighbours) by plane masks, and the
// 8-bit random-versus-threshold comparison by a bit-serial borrow chain.
//
// Randomness: the top byte of a site's acceptance word is bit-sliced -- eight
// planes from two Philox4x32-10 blocks per 32 sites (accept_word in
// common.cuh) -- so the planes of a word are exactly the kernel's operands.  The
// decision u53 < T(class) is taken on the top byte; a tie with the
// threshold's top byte (probability 1/256) is resolved with the site's fine
// block.  The result equals update_accepted<1>(dE, beta, word) bit for bit.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>
#include <cstring>

#include <cstdio>

#include "engine.h"

namespace mqv {

struct Ising2DArgs {
    const int8_t* src;
    int8_t* dst;
    int L;
    int ntx;
    int ntiles;
    Key key;
    uint32_t sweep;
    uint32_t replica;
    // The two aligned-neighbour classes with dE > 0: mode 0 (J < 0) tests
    // a = 3 (class A, dE = -4J) and a = 4 (class B, dE = -8J); mode 1 (J > 0)
    // tests a = 1 (A, dE = 4J) and a = 0 (B, dE = 8J); mode 2: no test.
    int mode;
    uint32_t useA, useB;        // 1 when the class needs a test (cut below 2^53)
    uint32_t tA8, tB8;          // threshold top bytes
    unsigned long long tA, tB;  // full u53 thresholds
    long long* acc;
    int* status;
    int* counter;  // next tile (zeroed before the launch)
    uint32_t rk0[10], rk1[10];  // Philox round keys of `key`
    // bounded waits: a wait gives up after wait_ns and sets MQV_ERR_TIMEOUT.
    // withhold >= 0 (tests of that path, band kernel only): CTA 0 never
    // issues its staged row `withhold`, so the wait for it runs out.
    unsigned long long wait_ns;
    int withhold;
};

// Philox4x32-10 with the round keys taken from the launch arguments (the
// same function as philox() in common.cuh, whose key schedule is computed
// once on the host)
__device__ __forceinline__ uint4 philox_rk(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, const Ising2DArgs& a)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        uint32_t hi0, lo0, hi1, lo1;
        mulhilo(0xD2511F53u, c0, hi0, lo0);
        mulhilo(0xCD9E8D57u, c2, hi1, lo1);
        const uint32_t n0 = hi1 ^ c1 ^ a.rk0[r];
        const uint32_t n2 = hi0 ^ c3 ^ a.rk1[r];
        c0 = n0;
        c1 = lo1;
        c2 = n2;
        c3 = lo0;
    }
    return make_uint4(c0, c1, c2, c3);
}

// low 56 bits of the acceptance word of `site` (accept_fine56 of common.cuh)
__device__ __forceinline__ uint64_t fine56_rk(uint32_t site, const Ising2DArgs& a)
{
    const uint4 f = philox_rk(site >> 1, a.sweep, 0u, (kAcceptFine << 24) | (a.replica & 0xFFFFFFu), a);
    return ((site & 1u) ? hi64(f) : lo64(f)) & 0x00FFFFFFFFFFFFFFull;
}

template <int TX, int TY, int NWARP>
struct TileGeom {
    static constexpr int NWI = TX / 64;         // interior 32-site words per half-row
    static constexpr int NWB = NWI + 2;         // with one halo word on each side
    static constexpr int H2 = TX / 2;           // interior sites per half-row
    static constexpr int PH = NWB * 32;         // staged bytes per half-row
    static constexpr int P = 2 * PH;            // staged bytes per row
    static constexpr int R = TY + 4;            // staged rows y0-2 .. y0+TY+1
    static constexpr int NS = 8;                // staging ring rows
    static constexpr int RPG = 32 / NWI;        // rows per 32 colour-1 words
    static constexpr int NO = 2 * RPG;          // output ring rows (two store groups)
    static constexpr int BITS = R * 2 * NWB * 4;
    static constexpr int STAGE = NS * P;
    static constexpr int OUT = NO * TX;
    static constexpr int TIECAP = 96;           // tie-list entries
    static constexpr int WARP = ((STAGE + OUT + BITS + NS * 8 + TIECAP * 20) + 127) / 128 * 128;  // per-warp partition
    static constexpr int SMEM = NWARP * WARP;
    static_assert(R % 4 == 0 && 32 % NWI == 0, "tile shape");
};

__device__ __forceinline__ int wrapi(int v, int L)
{
    v += v < 0 ? L : 0;
    return v >= L ? v - L : v;
}

// Per-launch constants of the decision, as all-ones / all-zeros lane masks.
struct Thr {
    uint32_t tA[8], tB[8];  // bit b of the class thresholds' top bytes
    uint32_t useA, useB;
    uint32_t anti;  // J > 0
};

__device__ __forceinline__ Thr make_thr(const Ising2DArgs& a)
{
    Thr t;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        t.tA[b] = 0u - ((a.tA8 >> b) & 1u);
        t.tB[b] = 0u - ((a.tB8 >> b) & 1u);
    }
    t.useA = a.mode == 2 ? 0u : 0u - a.useA;
    t.useB = a.mode == 2 ? 0u : 0u - a.useB;
    t.anti = a.mode == 1 ? ~0u : 0u;
    return t;
}

// A word whose tested sites include top-byte ties is recorded in the warp's
// tie list and resolved after the pass: a tie site's top byte equals its
// class threshold's top byte, so only its fine block is needed.
struct TieEntry {
    uint32_t pos;    // word position in the bit tile: (r * 2 + half) * NWB + w
    uint32_t tie;    // tie sites of the word
    uint32_t inA;    // tie sites of class A (others are class B)
    int32_t y, x;    // lattice coordinates of the word's first site
};

// The eight random planes of the word whose first site is (x, y): the two
// ACCEPT blocks of its 32-site group.
struct Planes {
    uint32_t b[8];
};
__device__ __forceinline__ Planes word_planes(int x, int y, uint32_t tg_acc, const Ising2DArgs& a)
{
    const uint32_t g = accept_group((uint32_t)y * (uint32_t)a.L + (uint32_t)x);
    const uint4 q0 = philox_rk(g, a.sweep, 0u, tg_acc, a);
    const uint4 q1 = philox_rk(g, a.sweep, 1u, tg_acc, a);
    return Planes{{q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w}};
}

// Update the active-colour sites of one 32-site word on its planes: returns
// the word with the decided flips applied; `tie` and `inA` receive the
// undecided sites.
__device__ __forceinline__ uint32_t decide_word(uint32_t A, uint32_t U, uint32_t D, uint32_t Lb, uint32_t Rb,
                                                const Planes& rnd, const Thr& th, uint32_t& tie, uint32_t& inA)
{
    const uint32_t* pl = rnd.b;
    // The tested classes count unlike neighbours: none (class B) and one (class
    // A) for J < 0, four and three for J > 0, which is the same of the flipped
    // site.  Carry-save adder of three neighbours plus the fourth; a majority
    // is self-dual, so comparing with the site comes after adding.
    const uint32_t S = A ^ th.anti;
    const uint32_t s3 = U ^ D ^ Lb, c3 = (U & D) | (Lb & (U | D));
    const uint32_t maskA = (s3 ^ Rb) & ~(c3 ^ S);
    const uint32_t maskB = ~((s3 ^ S) | (c3 ^ S)) & ~(Rb ^ S);
    const uint32_t test = (maskA & th.useA) | (maskB & th.useB);
    // X < T and X == T for the per-site threshold byte T (class A or B)
    uint32_t borrow = 0u, eq = test;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const uint32_t tb = (maskA & th.tA[b]) | (~maskA & th.tB[b]);
        const uint32_t nx = ~pl[b];
        borrow = (nx & (tb | borrow)) | (tb & borrow);
        eq &= ~(pl[b] ^ tb);
    }
    tie = eq;
    inA = eq & maskA;
    return A ^ (~test | borrow);
}
__device__ __forceinline__ uint32_t update_word(uint32_t A, uint32_t U, uint32_t D, uint32_t Lb, uint32_t Rb, int x,
                                                int y, uint32_t tg_acc, const Ising2DArgs& a, const Thr& th,
                                                uint32_t& tie, uint32_t& inA)
{
    return decide_word(A, U, D, Lb, Rb, word_planes(x, y, tg_acc, a), th, tie, inA);
}

// Bond sum s * sum(nbrs) = sum (1 - 2a)(4 - 2M) over the sites of a word
__device__ __forceinline__ int word_bonds(uint32_t An, uint32_t U, uint32_t D, uint32_t Lb, uint32_t Rb)
{
    const uint32_t s3 = U ^ D ^ Lb, c3 = (U & D) | (Lb & (U | D));  // full adder of three
    const uint32_t m0 = s3 ^ Rb, c4 = s3 & Rb;                        // plus the fourth
    const uint32_t m1 = c3 ^ c4, m2 = c3 & c4;
    const int sM = __popc(m0) + 2 * __popc(m1) + 4 * __popc(m2);
    const int sAM = __popc(An & m0) + 2 * __popc(An & m1) + 4 * __popc(An & m2);
    return 128 - 2 * sM - 8 * __popc(An) + 4 * sAM;
}

// 32 bits -> 32 bytes at p (16-byte aligned)
__device__ __forceinline__ void unpack32(uint32_t bits, uint8_t* p)
{
    uint4 lo, hi;
    unpack_word(bits, lo, hi);
    *reinterpret_cast<uint4*>(p) = lo;
    *reinterpret_cast<uint4*>(p + 16) = hi;
}

template <int TX, int TY, int NWARP, bool MEAS>
__global__ void __launch_bounds__(NWARP * 32) ising2d_sweep(const __grid_constant__ Ising2DArgs a)
{
    using G = TileGeom<TX, TY, NWARP>;
    constexpr int NWI = G::NWI, NWB = G::NWB, R = G::R, NS = G::NS;
    extern __shared__ __align__(128) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t* part = smem + warp * G::WARP;
    uint8_t* stage = part;                                                   // [NS][2][PH]
    uint8_t* out = part + G::STAGE;                                          // [NO][2][H2]
    uint32_t* bits = reinterpret_cast<uint32_t*>(part + G::STAGE + G::OUT);  // [R][2][NWB]
    uint64_t* bars = reinterpret_cast<uint64_t*>(part + G::STAGE + G::OUT + G::BITS);
    const int L = a.L, Lh = L >> 1;
    const uint32_t tg_acc = tag(kAccept, a.replica);
    const Thr th = make_thr(a);
    if (lane == 0) {
        for (int k = 0; k < NS; ++k) mbar_init(smem_addr(&bars[k]), 1);
        mbar_fence_init();
    }
    __syncwarp();

    // staged row q of this warp's row sequence (row r of tile `tile`) lands in
    // slot q % NS: the slot's byte count is armed once, then the copies of one
    // half-row are issued by the calling lane
    auto arm_row = [&](int q) { mbar_expect_tx(smem_addr(&bars[q % NS]), (uint32_t)G::P); };
    auto copy_half = [&](int tile, int r, int q, int h) {
        const int x0 = (tile % a.ntx) * TX, y0 = (tile / a.ntx) * TY;
        const uint32_t bar = smem_addr(&bars[q % NS]);
        const int8_t* rh = a.src + (size_t)wrapi(y0 - 2 + r, L) * L + (size_t)h * Lh;
        const uint32_t d = smem_addr(stage + (q % NS) * G::P + h * G::PH);
        const int j0 = (x0 >> 1) - 32;
        if (x0 > 0 && x0 + TX < L) {
            bulk_g2s(d, rh + j0, G::PH, bar);
        } else {
            bulk_g2s(d, rh + (j0 < 0 ? j0 + Lh : j0), 32, bar);
            bulk_g2s(d + 32, rh + (x0 >> 1), G::H2, bar);
            const int jr = (x0 >> 1) + G::H2;
            bulk_g2s(d + 32 + G::H2, rh + (jr >= Lh ? jr - Lh : jr), 32, bar);
        }
    };
    // rows q0 .. q0+n-1 (rows r0.. of `tile`, continuing into `tile2` past R):
    // lanes 0..n-1 arm, lanes 0..2n-1 copy one half-row each
    auto issue_rows = [&](int tile, int tile2, int r0, int q0, int n) {
        if (lane < n) {
            const int r = r0 + lane;
            if (r < R || tile2 < a.ntiles) arm_row(q0 + lane);
        }
        __syncwarp();
        if (lane < 2 * n) {
            const int i = lane >> 1, r = r0 + i;
            if (r < R) copy_half(tile, r, q0 + i, lane & 1);
            else if (tile2 < a.ntiles) copy_half(tile2, r - R, q0 + i, lane & 1);
        }
    };
    auto grab = [&]() {
        int t = 0;
        if (lane == 0) t = atomicAdd(a.counter, 1);
        return __shfl_sync(0xffffffffu, t, 0);
    };

    // the warp's tie list: entries appended with a ballot, resolved in bulk
    TieEntry* tl = reinterpret_cast<TieEntry*>(part + G::STAGE + G::OUT + G::BITS + NS * 8);
    int ntie = 0;
    auto flush_ties = [&]() {
        __syncwarp();
        for (int e = lane; e < ntie; e += 32) {
            const TieEntry t = tl[e];
            uint32_t m = t.tie, flips = 0u;
            while (m) {
                const int b = __ffs(m) - 1;
                m &= m - 1;
                const bool inA = (t.inA >> b) & 1u;
                const uint32_t site = (uint32_t)t.y * (uint32_t)L + (uint32_t)(t.x + 2 * b);
                const uint64_t u53 = ((uint64_t)(inA ? a.tA8 : a.tB8) << 45) |
                                     (fine56_rk(site, a) >> 11);
                if (u53 < (inA ? a.tA : a.tB)) flips |= 1u << b;
            }
            if (flips) bits[t.pos] ^= flips;
        }
        __syncwarp();
        ntie = 0;
    };
    auto record_ties = [&](uint32_t tie, uint32_t inA, uint32_t pos, int yy, int xx) {
        const uint32_t has = __ballot_sync(0xffffffffu, tie != 0u);
        if (tie) tl[ntie + __popc(has & ((1u << lane) - 1u))] = TieEntry{pos, tie, inA, yy, xx};
        ntie += __popc(has);
        if (ntie > G::TIECAP - 32) flush_ties();
    };

    int esum = 0, msum = 0;
    uint32_t gq = 0;  // store groups issued by this warp: output-ring half = gq & 1
    int cur = grab();
    int nxt = cur < a.ntiles ? grab() : a.ntiles;
    int base = 0;  // sequence number of the current tile's row 0
    if (cur < a.ntiles) {
        fence_proxy_async_smem();
        issue_rows(cur, a.ntiles, 0, 0, NS);
    }
    bool stop = false;
    while (cur < a.ntiles && !stop) {
        const int x0 = (cur % a.ntx) * TX, y0 = (cur / a.ntx) * TY;
        // stream the staged rows in, four at a time, packing them to bits
        for (int r0 = 0; r0 < R; r0 += 4) {
            // every lane waits for the four rows (bounded: a stuck copy sets an error status)
            int timed_out = 0;
            for (int i = 0; i < 4 && !timed_out; ++i) {
                const int q = base + r0 + i;
                const uint32_t bar = smem_addr(&bars[q % NS]);
                const uint32_t par = (uint32_t)(q / NS) & 1u;
                if (!mbar_try_wait(bar, par)) {
                    // back off so that waiting warps leave their issue slots to others
                    const uint64_t t0 = global_timer_ns();
                    for (uint32_t k = 1;; ++k) {
                        __nanosleep(64);
                        if (mbar_try_wait(bar, par)) break;
                        if ((k & 63u) == 0 && global_timer_ns() - t0 > a.wait_ns) {
                            timed_out = 1;
                            break;
                        }
                    }
                }
            }
            if (__any_sync(0xffffffffu, timed_out)) {
                if (lane == 0) atomicExch(a.status, MQV_ERR_TIMEOUT);
                stop = true;
                break;
            }
            // 4 rows x 2 halves x NWB words = 8 NWB words = 16 NWB chunks of 16 bytes
            for (int c0 = 0; c0 < 16 * NWB; c0 += 32) {
                const int c = c0 + lane;
                uint32_t h16 = 0;
                if (c < 16 * NWB) {
                    const int i = c / (4 * NWB), cr = c % (4 * NWB);
                    const uint8_t* sb = stage + ((base + r0 + i) % NS) * G::P;
                    h16 = pack_lanes4(reinterpret_cast<const uint4*>(sb)[cr]) << (4 * (c & 1));
                }
                const uint32_t hi = __shfl_down_sync(0xffffffffu, h16, 1);
                if (!(c & 1) && c < 16 * NWB) bits[(r0 * 2 * NWB) + (c >> 1)] = h16 | hi;
            }
            __syncwarp();
            // refill the four freed slots: rows NS ahead in this tile or the next
            fence_proxy_async_smem();
            issue_rows(cur, nxt, r0 + NS, base + r0 + NS, 4);
        }
        if (stop) break;
        __syncwarp();
        // colour 0 on the tile and its ring: rows 1..TY+2, interior words + one halo word
        for (int t0 = 0; t0 < (TY + 2) * (NWI + 1); t0 += 32) {
            const int task = t0 + lane;
            uint32_t tie = 0u, inA = 0u, pos = 0u;
            int yy = 0, xx = 0;
            if (task < (TY + 2) * (NWI + 1)) {
                const int r = 1 + task / (NWI + 1), k = task % (NWI + 1);
                const int p = r & 1;
                const int w = k < NWI ? 1 + k : (p ? 0 : NWI + 1);
                pos = (uint32_t)((r * 2 + p) * NWB + w);
                const uint32_t* Gr = bits + (r * 2 + (1 - p)) * NWB;
                const uint32_t Gw = Gr[w];
                const uint32_t Lb = p ? Gw : __funnelshift_l(Gr[w - 1], Gw, 1);
                const uint32_t Rb = p ? __funnelshift_r(Gw, Gr[w + 1], 1) : Gw;
                yy = wrapi(y0 - 2 + r, L);
                xx = wrapi(x0 - 64 + 64 * w + p, L);
                bits[pos] = update_word(bits[pos], bits[pos - 2 * NWB], bits[pos + 2 * NWB], Lb, Rb, xx, yy, tg_acc,
                                        a, th, tie, inA);
            }
            record_ties(tie, inA, pos, yy, xx);
        }
        flush_ties();
        // colour 1 on the tile
        for (int t0 = 0; t0 < TY * NWI; t0 += 32) {
            const int task = t0 + lane;
            const int r = 2 + task / NWI, w = 1 + task % NWI;
            const int p = (r + 1) & 1;
            const uint32_t pos = (uint32_t)((r * 2 + p) * NWB + w);
            const uint32_t* Gr = bits + (r * 2 + (1 - p)) * NWB;
            const uint32_t Gw = Gr[w];
            const uint32_t Lb = p ? Gw : __funnelshift_l(Gr[w - 1], Gw, 1);
            const uint32_t Rb = p ? __funnelshift_r(Gw, Gr[w + 1], 1) : Gw;
            const int yy = wrapi(y0 - 2 + r, L), xx = wrapi(x0 - 64 + 64 * w + p, L);
            uint32_t tie, inA;
            bits[pos] = update_word(bits[pos], bits[pos - 2 * NWB], bits[pos + 2 * NWB], Lb, Rb, xx, yy, tg_acc, a,
                                    th, tie, inA);
            record_ties(tie, inA, pos, yy, xx);
        }
        flush_ties();
        // the tile's rows to the output ring and out, RPG rows (32 words) at a time
        for (int t0 = 0; t0 < TY * NWI; t0 += 32) {
            const int task = t0 + lane;
            const int r = 2 + task / NWI, w = 1 + task % NWI;
            const int p = (r + 1) & 1;
            const uint32_t pos = (uint32_t)((r * 2 + p) * NWB + w);
            const uint32_t* Gr = bits + (r * 2 + (1 - p)) * NWB;
            const uint32_t An = bits[pos], Gw = Gr[w];
            if (MEAS) {
                const uint32_t Lb = p ? Gw : __funnelshift_l(Gr[w - 1], Gw, 1);
                const uint32_t Rb = p ? __funnelshift_r(Gw, Gr[w + 1], 1) : Gw;
                esum += word_bonds(An, bits[pos - 2 * NWB], bits[pos + 2 * NWB], Lb, Rb);
                msum += 64 - 2 * __popc(An) - 2 * __popc(Gw);
            }
            // the output-ring half this group uses must have been read by its
            // last stores (each storing lane waits for its own bulk groups)
            if (lane < 2 * G::RPG) bulk_wait_read1();
            __syncwarp();
            uint8_t* orow = out + ((gq & 1u) * G::RPG + lane / NWI) * TX;
            unpack32(An, orow + p * G::H2 + 32 * (w - 1));
            unpack32(Gw, orow + (1 - p) * G::H2 + 32 * (w - 1));
            fence_proxy_async_smem();
            __syncwarp();
            if (lane < 2 * G::RPG) {
                for (int k = lane; k < 2 * G::RPG; k += 32) {
                    const int i = k >> 1, h = k & 1;
                    const int rr = 2 + t0 / NWI + i;
                    const uint8_t* src = out + ((gq & 1u) * G::RPG + i) * TX + h * G::H2;
                    int8_t* drow = a.dst + (size_t)(y0 + rr - 2) * L + (size_t)h * Lh + (x0 >> 1);
                    bulk_s2g(drow, smem_addr(src), G::H2);
                }
                bulk_commit();
            }
            ++gq;
        }
        base += R;
        cur = nxt;
        nxt = cur < a.ntiles ? grab() : a.ntiles;
    }
    bulk_wait0();
    if (MEAS) {
        long long e = esum, m = msum;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            e += __shfl_xor_sync(0xffffffffu, e, o);
            m += __shfl_xor_sync(0xffffffffu, m, o);
        }
        if (lane == 0) {
            // enepart = sum_i sum_{j in nbrs(i)} s_i s_j counts every bond twice
            atomicAdd(reinterpret_cast<unsigned long long*>(a.acc + kAccEne), (unsigned long long)(2 * e));
            atomicAdd(reinterpret_cast<unsigned long long*>(a.acc + kAccMag), (unsigned long long)m);
        }
    }
}

// ---- band kernel: one CTA spans the lattice width --------------------------------
//
// Thread t owns word columns t, t + NT, ..., t + (W - 1) NT of both halves of
// every row (64 sites each: 32 even-x and 32 odd-x), so a CTA of L / (64 W)
// threads covers whole rows and needs no horizontal halo.  CTA c streams down its band of rows [y0, y1) (bands split
// the L rows evenly over the grid) with two halo rows above and below: staged
// row r is lattice row y0 - 2 + r, r = 0 .. H + 3.  Step k of the pipeline
//   packs staged row k (one bulk copy per row, ring of NSB slots) into the bit
//   ring, updates colour 0 of row k - 1, colour 1 of row k - 2 - S, and writes
//   row k - 2 - 2S out.
// Top-byte ties of both colours are resolved in bulk every S steps, so a word
// is final at most S - 1 steps after its update: colour 1 lags colour 0 by S
// rows and the output lags colour 1 by S rows, which keeps every neighbour a
// word reads final.  The bit ring keeps the last RB = 2S + 4 rows.  With
// W > 1 a thread carries W independent words through every stage of a step.

template <int NT, int S, int NSB_, int W = 1>  // NT threads of W columns; ties every S steps; NSB_ staged rows
struct BandGeom {
    static constexpr int NW = NT / 32;
    static constexpr int NC = NT * W;            // word columns
    static constexpr int NSB = NSB_;             // staged row slots
    static constexpr int RB = 2 * S + 4;         // bit ring rows
    static constexpr int L = NC * 64;
    static constexpr int STAGE = NSB * L;
    static constexpr int BITS = RB * 2 * NC * 4;
    static constexpr int TIECAP = 32 + 64 * W;   // tie entries per warp: a step adds at most 64 W
    static constexpr int TIES = NW * TIECAP * 16;
    static constexpr int SMEM = STAGE + BITS + TIES + NSB * 8;
    static constexpr int SMEM_RS = BITS + TIES;  // register-staged rows: no staging ring
    static_assert(NT % 32 == 0 && S >= 1 && W >= 1, "band shape");
};

struct BandTie {
    uint32_t pos;  // word position in the bit ring: (slot * 2 + half) * NC + column
    uint32_t tie;  // undecided sites of the word
    uint32_t inA;  // those of class A
    int32_t y;     // lattice row
};

// RS (register staging): instead of the bulk-copy ring, every thread loads
// its own columns of staged row k + 1 into registers (two 16-byte loads per
// column and half, a warp's loads one contiguous kilobyte) right after packing
// row k, so the loads are in flight during the step's updates and are packed
// after the next barrier.  Without the staging ring a CTA needs a third of the
// shared memory, and more CTAs share an SM; no wait can hang (plain loads).
// MINB: CTAs per SM the register allocation must allow (0: no bound).
template <int NT, int S, int NSB_, bool MEAS, int W = 1, bool RS = false, int MINB = 0>
__global__ void __launch_bounds__(NT, MINB) ising2d_band(const __grid_constant__ Ising2DArgs a)
{
    using G = BandGeom<NT, S, NSB_, W>;
    constexpr int RB = G::RB, NSB = G::NSB, L = G::L, Lh = L / 2, NC = G::NC;
    constexpr int STAGE = RS ? 0 : G::STAGE;
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* stage = smem;
    uint32_t* bits = reinterpret_cast<uint32_t*>(smem + STAGE);
    BandTie* ties = reinterpret_cast<BandTie*>(smem + STAGE + G::BITS);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGE + G::BITS + G::TIES);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int y0 = (int)(((long long)blockIdx.x * L) / gridDim.x);
    const int y1 = (int)(((long long)(blockIdx.x + 1) * L) / gridDim.x);
    const int NR = y1 - y0 + 4;  // staged rows
    const uint32_t tg_acc = tag(kAccept, a.replica);
    const Thr th = make_thr(a);
    // column of word j of this thread, and the left / right neighbour columns
    auto col = [&](int j) { return t + j * NT; };
    auto coll = [&](int c) { return c == 0 ? NC - 1 : c - 1; };
    auto colr = [&](int c) { return c == NC - 1 ? 0 : c + 1; };

    if (!RS && t == 0) {
        for (int k = 0; k < NSB; ++k) mbar_init(smem_addr(&bars[k]), 1);
        mbar_fence_init();
    }
    __syncthreads();
    // staged row r -> slot r % NSB (thread 0)
    auto issue = [&](int r) {
        if (blockIdx.x == 0 && r == a.withhold) return;  // injected: the row's wait runs out
        const int y = wrapi(y0 - 2 + r, L);
        const uint32_t bar = smem_addr(&bars[r % NSB]);
        mbar_expect_tx(bar, (uint32_t)L);
        bulk_g2s(smem_addr(stage + (r % NSB) * L), a.src + (size_t)y * L, (uint32_t)L, bar);
    };
    if (!RS && t == 0)
        for (int r = 0; r < NSB && r < NR; ++r) issue(r);
    // RS: this thread's bytes of the next staged row, [column][half][16-byte part]
    uint4 pre[RS ? W : 1][2][2];
    auto load_row = [&](int r) {
        const int8_t* rowp = a.src + (size_t)wrapi(y0 - 2 + r, L) * L;
#pragma unroll
        for (int j = 0; j < W; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4* q = reinterpret_cast<const uint4*>(rowp + h * Lh + 32 * col(j));
                pre[RS ? j : 0][h][0] = __ldg(q);
                pre[RS ? j : 0][h][1] = __ldg(q + 1);
            }
    };
    if (RS) load_row(0);

    BandTie* tl = ties + warp * G::TIECAP;
    int ntie = 0;
    auto record = [&](uint32_t tie, uint32_t inA, uint32_t pos, int y) {
        const uint32_t has = __ballot_sync(0xffffffffu, tie != 0u);
        if (tie) tl[ntie + __popc(has & ((1u << lane) - 1u))] = BandTie{pos, tie, inA, y};
        ntie += __popc(has);
    };
    auto flush = [&]() {
        __syncwarp();
        for (int e = lane; e < ntie; e += 32) {
            const BandTie te = tl[e];
            const uint32_t w = te.pos % NC, h = (te.pos / NC) & 1u;
            const uint32_t site0 = (uint32_t)te.y * (uint32_t)L + 64u * w + h;
            uint32_t m = te.tie, flips = 0u;
            while (m) {
                const int b = __ffs(m) - 1;
                m &= m - 1;
                const bool inA = (te.inA >> b) & 1u;
                const uint64_t u53 = ((uint64_t)(inA ? a.tA8 : a.tB8) << 45) |
                                     (fine56_rk(site0 + 2u * (uint32_t)b, a) >> 11);
                if (u53 < (inA ? a.tA : a.tB)) flips |= 1u << b;
            }
            if (flips) bits[te.pos] ^= flips;
        }
        __syncwarp();
        ntie = 0;
    };
    // inputs of the word of column c in half p of staged row r
    struct WordIn {
        uint32_t A, U, D, Lb, Rb, pos;
    };
    auto word_in = [&](int sl, int su, int sd, int p, int c) {
        WordIn w;
        w.pos = (uint32_t)((sl * 2 + p) * NC + c);
        const uint32_t* Gr = bits + (sl * 2 + (1 - p)) * NC;
        const uint32_t Gw = Gr[c];
        w.Lb = p ? Gw : __funnelshift_l(Gr[coll(c)], Gw, 1);
        w.Rb = p ? __funnelshift_r(Gw, Gr[colr(c)], 1) : Gw;
        w.A = bits[w.pos];
        w.U = bits[(su * 2 + p) * NC + c];
        w.D = bits[(sd * 2 + p) * NC + c];
        return w;
    };
    // update this thread's words in half p of staged row r (lattice row y)
    auto update = [&](int sl, int su, int sd, int p, int y) {
#pragma unroll
        for (int j = 0; j < W; ++j) {
            const int c = col(j);
            const WordIn w = word_in(sl, su, sd, p, c);
            uint32_t tie, inA;
            bits[w.pos] = update_word(w.A, w.U, w.D, w.Lb, w.Rb, 64 * c + p, y, tg_acc, a, th, tie, inA);
            record(tie, inA, w.pos, y);
        }
    };

    int esum = 0, msum = 0;
    int k = 0;
    int sk = 0;  // k % RB: the bit-ring slot of staged row k
    // slot of staged row k - d (0 <= d < RB)
    auto back = [&](int d) {
        const int v = sk - d;
        return v < 0 ? v + RB : v;
    };
    bool stop = false;
    for (; k < NR + 2 * S; ++k, sk = sk + 1 == RB ? 0 : sk + 1) {
        int timed_out = 0;
        if (!RS && k < NR) {
            // every thread waits for row k (bounded: a stuck copy sets an error status)
            const uint32_t bar = smem_addr(&bars[k % NSB]);
            const uint32_t par = (uint32_t)(k / NSB) & 1u;
            if (!mbar_try_wait(bar, par)) {
                const uint64_t t0 = global_timer_ns();
                for (uint32_t i = 1;; ++i) {
                    __nanosleep(64);
                    if (mbar_try_wait(bar, par)) break;
                    if ((i & 63u) == 0 && global_timer_ns() - t0 > a.wait_ns) {
                        timed_out = 1;
                        break;
                    }
                }
            }
        }
        // one barrier per step: the previous step's words are visible to their
        // readers, and every warp has packed row k - 1, so its slot is free
        if (__syncthreads_or(timed_out)) {
            stop = true;
            break;
        }
        if (!RS && t == 0 && k >= 1 && k - 1 + NSB < NR) {
            fence_proxy_async_smem();
            issue(k - 1 + NSB);
        }
        if (k < NR) {
            uint32_t* brow = bits + sk * 2 * NC;
            if (RS) {
#pragma unroll
                for (int j = 0; j < W; ++j)
#pragma unroll
                    for (int h = 0; h < 2; ++h) brow[h * NC + col(j)] = pack_word(pre[RS ? j : 0][h][0], pre[RS ? j : 0][h][1]);
                if (k + 1 < NR) load_row(k + 1);
            } else {
                const uint8_t* row = stage + (k % NSB) * L;
#pragma unroll
                for (int j = 0; j < W; ++j) {
                    const int c = col(j);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint4* q = reinterpret_cast<const uint4*>(row + h * Lh + 32 * c);
                        brow[h * NC + c] = pack_word(q[0], q[1]);
                    }
                }
            }
        }
        // row k's bits are read in this step only by their own thread (the D
        // neighbour of colour 0 in row k - 1); other warps read them from the
        // next step on, after its barrier
        // colour 0 of row k - 1 (staged rows 1 .. NR - 2) and colour 1 of row
        // k - 2 - S (staged rows 2 .. NR - 3): independent words, updated
        // side by side in the steady state
        const int r1 = k - 2 - S;
        const bool do0 = k - 1 >= 1 && k - 1 <= NR - 2, do1 = r1 >= 2 && r1 <= NR - 3;
        const int ya = wrapi(y0 - 3 + k, L), yb = y0 - 2 + r1;
        if (do0 && do1) {
            const int pa = ya & 1, pb = 1 - (yb & 1);
#pragma unroll
            for (int j = 0; j < W; ++j) {
                const int c = col(j);
                const WordIn wa = word_in(back(1), back(2), sk, pa, c);
                const WordIn wb = word_in(back(2 + S), back(3 + S), back(1 + S), pb, c);
                uint32_t ta, ia, tb, ib;
                const uint32_t na =
                    update_word(wa.A, wa.U, wa.D, wa.Lb, wa.Rb, 64 * c + pa, ya, tg_acc, a, th, ta, ia);
                const uint32_t nb =
                    update_word(wb.A, wb.U, wb.D, wb.Lb, wb.Rb, 64 * c + pb, yb, tg_acc, a, th, tb, ib);
                bits[wa.pos] = na;
                bits[wb.pos] = nb;
                record(ta, ia, wa.pos, ya);
                record(tb, ib, wb.pos, yb);
            }
        } else if (do0) {
            update(back(1), back(2), sk, ya & 1, ya);
        } else if (do1) {
            update(back(2 + S), back(3 + S), back(1 + S), 1 - (yb & 1), yb);
        }
        if (k % S == S - 1 || ntie > G::TIECAP - 64 * W) flush();
        // row k - 2 - 2S out
        const int r2 = k - 2 - 2 * S;
        if (r2 >= 2 && r2 <= NR - 3) {
            const int y = y0 - 2 + r2;
            const int sl = back(2 + 2 * S);
#pragma unroll
            for (int j = 0; j < W; ++j) {
                const int c = col(j);
                const uint32_t w0 = bits[(sl * 2) * NC + c], w1 = bits[(sl * 2 + 1) * NC + c];
                int8_t* drow = a.dst + (size_t)y * L + 32 * c;
                uint4 lo, hi;
                unpack_word(w0, lo, hi);
                reinterpret_cast<uint4*>(drow)[0] = lo;
                reinterpret_cast<uint4*>(drow)[1] = hi;
                unpack_word(w1, lo, hi);
                reinterpret_cast<uint4*>(drow + Lh)[0] = lo;
                reinterpret_cast<uint4*>(drow + Lh)[1] = hi;
                if (MEAS) {
                    const int p1 = 1 - (y & 1);
                    const uint32_t An = p1 ? w1 : w0, Gw = p1 ? w0 : w1;
                    const uint32_t* Gr = bits + (sl * 2 + (1 - p1)) * NC;
                    const uint32_t Lb = p1 ? Gw : __funnelshift_l(Gr[coll(c)], Gw, 1);
                    const uint32_t Rb = p1 ? __funnelshift_r(Gw, Gr[colr(c)], 1) : Gw;
                    const uint32_t U = bits[(back(3 + 2 * S) * 2 + p1) * NC + c];
                    const uint32_t D = bits[(back(1 + 2 * S) * 2 + p1) * NC + c];
                    esum += word_bonds(An, U, D, Lb, Rb);
                    msum += 64 - 2 * __popc(An) - 2 * __popc(Gw);
                }
            }
        }
    }
    if (stop) {
        // wait (bounded) for the copies still in flight before the CTA leaves
        if (!RS && t == 0) {
            atomicExch(a.status, MQV_ERR_TIMEOUT);
            const uint64_t t0 = global_timer_ns();
            const int issued = k == 0 ? NSB : k - 1 + NSB;  // rows issued before the stop
            for (int r = k; r < NR && r < issued; ++r) {
                if (blockIdx.x == 0 && r == a.withhold) continue;  // never issued
                const uint32_t bar = smem_addr(&bars[r % NSB]);
                const uint32_t par = (uint32_t)(r / NSB) & 1u;
                while (!mbar_try_wait(bar, par) && global_timer_ns() - t0 < 1000000000ull) __nanosleep(1000);
            }
        }
        return;
    }
    if (MEAS) {
        long long e = esum, m = msum;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            e += __shfl_xor_sync(0xffffffffu, e, o);
            m += __shfl_xor_sync(0xffffffffu, m, o);
        }
        if (lane == 0) {
            atomicAdd(reinterpret_cast<unsigned long long*>(a.acc + kAccEne), (unsigned long long)(2 * e));
            atomicAdd(reinterpret_cast<unsigned long long*>(a.acc + kAccMag), (unsigned long long)m);
        }
    }
}

// ---- colour kernel: one launch per colour, in place ------------------------------
//
// For lattices that fit the L2 (L <= 8192): thread = T consecutive rows of one
// word column.  A word of the colour needs its own 32 bytes and, from the rows
// above, here and below, the other colour's words of the same column plus one
// edge byte of the neighbouring column; a strip of T rows shares them, so a
// word update packs 2 + 2 / T words.  Sites of one colour are independent and
// only the active words are written, so the update is in place, without halo
// re-computation, barriers or a tile queue: what bounds it is the latency of a
// few dependent loads at small L and the instruction issue rate at large L
// (per sweep, before with tiles and now: L = 1024 37.6 -> 7 us, L = 4096 50.8
// -> 12.3 us; starting the draws before the previous launch has drained took
// them from 8.5 and 16.8 us).
// Top-byte ties are listed per warp and resolved after the strip, side by side
// over the lanes; an accepted one is stored as a byte.  MEAS (launched for
// colour 1): every bond joins a colour-1 site to a colour-0 site, so the
// colour-1 words' bond sums after the update are the lattice's.
template <int T>
struct ColourGeom {
    static constexpr int NT = 256;
    static constexpr int TIECAP = 32 * T;  // every word of the warp's strips may hold ties
};

template <int T, bool MEAS>
__global__ void __launch_bounds__(ColourGeom<T>::NT) ising2d_colour(const __grid_constant__ Ising2DArgs a, int colour)
{
    using G = ColourGeom<T>;
    __shared__ uint4 ties[G::NT / 32][G::TIECAP];  // (row ncol + column, tie sites, class A, word)
    __shared__ int red[2][G::NT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int L = a.L, Lh = L >> 1, ncol = L >> 6;
    const uint32_t nstrip = (uint32_t)ncol * (uint32_t)(L / T);
    const uint32_t id = blockIdx.x * G::NT + threadIdx.x;
    const bool live = id < nstrip;
    const uint32_t strip = live ? id : 0u, sy = strip / (uint32_t)ncol;
    const int w = (int)(strip - sy * (uint32_t)ncol), y0 = (int)sy * T;
    const uint32_t tg_acc = tag(kAccept, a.replica);
    const Thr th = make_thr(a);
    int8_t* s = a.dst;
    // the draws need no lattice data: they run while the launch before this
    // one drains (programmatic dependent launch), the state is touched after
    Planes rnd[T];
#pragma unroll
    for (int k = 0; k < T; ++k) rnd[k] = word_planes(64 * w + ((y0 + k + colour) & 1), y0 + k, tg_acc, a);
    grid_dep_launch();
    grid_dep_wait();
    // the other colour's words of rows y0 - 1 .. y0 + T (half 1 - p of a row
    // whose active half is p), the active words, the edge sites
    uint32_t g[T + 2], act[T], edge[T];
#pragma unroll
    for (int k = 0; k < T + 2; ++k) {
        const int y = wrapi(y0 - 1 + k, L), p = (y0 - 1 + k + colour) & 1;
        const int8_t* row = s + (size_t)y * L;
        const uint4* q = reinterpret_cast<const uint4*>(row + (p ? 0 : Lh) + 32 * w);
        g[k] = pack_word(q[0], q[1]);
        if (k >= 1 && k <= T) {
            const uint4* qa = reinterpret_cast<const uint4*>(row + (p ? Lh : 0) + 32 * w);
            act[k - 1] = pack_word(qa[0], qa[1]);
            // p = 1: site 0 of the even word to the right; p = 0: site 31 of the odd word to the left
            const int8_t e = p ? row[32 * (w + 1 == ncol ? 0 : w + 1)] : row[Lh + 32 * (w == 0 ? ncol - 1 : w - 1) + 31];
            edge[k - 1] = (uint32_t)e >> 31;
        }
    }
    int ntie = 0, esum = 0, msum = 0;
#pragma unroll
    for (int k = 0; k < T; ++k) {
        const int y = y0 + k, p = (y + colour) & 1;
        const uint32_t G1 = g[k + 1];
        const uint32_t Lb = p ? G1 : (G1 << 1) | edge[k];
        const uint32_t Rb = p ? (G1 >> 1) | (edge[k] << 31) : G1;
        uint32_t tie, inA;
        const uint32_t An = decide_word(act[k], g[k], g[k + 2], Lb, Rb, rnd[k], th, tie, inA);
        if (!live) tie = 0u;
        const uint32_t has = __ballot_sync(0xffffffffu, tie != 0u);
        if (tie)
            ties[warp][ntie + __popc(has & ((1u << lane) - 1u))] =
                make_uint4((uint32_t)y * (uint32_t)ncol + (uint32_t)w, tie, inA, An);
        ntie += __popc(has);
        if (live) {
            uint4 lo, hi;
            unpack_word(An, lo, hi);
            uint4* q = reinterpret_cast<uint4*>(s + (size_t)y * L + (p ? Lh : 0) + 32 * w);
            q[0] = lo;
            q[1] = hi;
            if (MEAS) {
                esum += word_bonds(An, g[k], g[k + 2], Lb, Rb);
                msum += 64 - 2 * __popc(An) - 2 * __popc(G1);
            }
        }
    }
    __syncwarp();
    for (int e = lane; e < ntie; e += 32) {
        const uint4 te = ties[warp][e];
        const uint32_t y = te.x / (uint32_t)ncol, c = te.x - y * (uint32_t)ncol, p = (y + (uint32_t)colour) & 1u;
        uint32_t m = te.y;
        while (m) {
            const int b = __ffs(m) - 1;
            m &= m - 1;
            const bool inA = (te.z >> b) & 1u;
            const uint64_t u53 = ((uint64_t)(inA ? a.tA8 : a.tB8) << 45) |
                                 (fine56_rk(y * (uint32_t)L + 64u * c + p + 2u * (uint32_t)b, a) >> 11);
            if (u53 < (inA ? a.tA : a.tB)) {
                const bool minus = (te.w >> b) & 1u;
                s[(size_t)y * L + (p ? Lh : 0) + 32 * c + 4 * (b & 7) + (b >> 3)] = minus ? 1 : -1;
                if (MEAS) {
                    // the tested classes have s * sum(nbrs) = +-2 (A) or +-4 (B) before the flip
                    esum += (inA ? 4 : 8) * (a.mode == 0 ? -1 : 1);
                    msum += minus ? 2 : -2;
                }
            }
        }
    }
    if (MEAS) {
        esum = __reduce_add_sync(0xffffffffu, esum);
        msum = __reduce_add_sync(0xffffffffu, msum);
        if (lane == 0) {
            red[0][warp] = esum;
            red[1][warp] = msum;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            long long e = 0, m = 0;
            for (int k = 0; k < G::NT / 32; ++k) {
                e += red[0][k];
                m += red[1][k];
            }
            atomicAdd(reinterpret_cast<unsigned long long*>(a.acc + kAccEne), (unsigned long long)(2 * e));
            atomicAdd(reinterpret_cast<unsigned long long*>(a.acc + kAccMag), (unsigned long long)m);
        }
    }
}

// ---- bit planes: several sweeps between two visits to the int8 state -------------
//
// A run of sweeps with nothing between them but measurements packs the state
// once into a bit per site (in the spare state buffer: row y holds the L/64
// words of its even half, then those of its odd half), sweeps the bits in
// place, a launch per colour, and unpacks at the end.  A word update then
// costs its draws and its logic and nothing else: no packing (30 of about 240
// instructions), 5 words of L2 traffic instead of 4 x 32 bytes of HBM (L =
// 16384: 34 MB of bits).  Bound by the ALU pipe (two Philox blocks, a
// carry-save adder and an 8-step comparison per 32 sites).  Thread = T rows of
// one word column, as in the colour kernel; the draws of its first rows come
// before the launch waits for its predecessor.
// Per sweep, int8 kernels before and this one (us): L = 1024 5.5 -> 4.0, L = 4096
// 12.1 -> 7.7, L = 8192 38.5 -> 21.2, L = 16384 114 -> 71; packing and unpacking
// together take what 1.4 sweeps take at L = 16384.  At L = 16384 186 instructions
// per word, half of them for the Philox blocks, the ALU pipe busy 63 % of the time.
template <int T>
struct BitsGeom {
    static constexpr int NT = T <= 2 ? 128 : 256;
    static constexpr int TIECAP = 32 * T;       // every word of the warp's strips may hold ties
    static constexpr int EARLY = T < 2 ? T : T <= 4 ? 2 : 0;  // rows whose draws come before the launch waits
};

__global__ void __launch_bounds__(256) ising2d_pack(const int8_t* __restrict__ s, uint32_t* __restrict__ bits,
                                                    int64_t words)
{
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= words) return;
    const uint4* q = reinterpret_cast<const uint4*>(s) + 2 * k;
    const uint4 lo = __ldcs(q), hi = __ldcs(q + 1);
    bits[k] = pack_word(lo, hi);
}
__global__ void __launch_bounds__(256) ising2d_unpack(const uint32_t* __restrict__ bits, int8_t* __restrict__ s,
                                                      int64_t words)
{
    grid_dep_wait();
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= words) return;
    uint4 lo, hi;
    unpack_word(bits[k], lo, hi);
    uint4* q = reinterpret_cast<uint4*>(s) + 2 * k;
    __stcs(q, lo);
    __stcs(q + 1, hi);
}

// sum over the sites of a word of s * sum(nbrs): 4 per site less 2 per unlike
// neighbour, the unlike neighbours added up by the carry-save adder
__device__ __forceinline__ int word_bonds_unlike(uint32_t An, uint32_t U, uint32_t D, uint32_t Lb, uint32_t Rb)
{
    U ^= An;
    D ^= An;
    Lb ^= An;
    Rb ^= An;
    const uint32_t s3 = U ^ D ^ Lb, c3 = (U & D) | (Lb & (U | D));
    const uint32_t m0 = s3 ^ Rb, c4 = s3 & Rb;
    return 128 - 2 * __popc(m0) - 4 * __popc(c3 ^ c4) - 8 * __popc(c3 & c4);
}

template <int T, int COLOUR, bool MEAS>
__global__ void __launch_bounds__(BitsGeom<T>::NT) ising2d_bits(const __grid_constant__ Ising2DArgs a)
{
    using G = BitsGeom<T>;
    __shared__ uint4 ties[G::NT / 32][G::TIECAP];         // (byte offset, tie sites, class A, word)
    __shared__ uint32_t tie_site[G::NT / 32][G::TIECAP];  // the word's first site
    __shared__ int red[2][G::NT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t L = (uint32_t)a.L, ncol = L >> 6, half = 4 * ncol, pitch = 8 * ncol;  // bytes of a half-row and row
    const uint32_t nstrip = ncol * (L / T);
    const uint32_t id = blockIdx.x * G::NT + threadIdx.x;
    const bool live = id < nstrip;
    const uint32_t strip = live ? id : 0u, sy = strip / ncol, w = strip - sy * ncol, y0 = sy * T;
    const uint32_t tg_acc = tag(kAccept, a.replica);
    Thr th = make_thr(a);
#pragma unroll
    for (int b = 0; b < 8; ++b) asm volatile("" : "+r"(th.tA[b]), "+r"(th.tB[b]));  // held, not derived again per word
    // parity of the active half of row y0 + k; a strip of an even number of
    // rows starts on an even one
    const uint32_t odd = T % 2 ? y0 & 1u : 0u;
    auto par = [&](int k) -> uint32_t { return ((uint32_t)(k + COLOUR) + odd) & 1u; };
    // the word's 32-site group (accept_group of its first site)
    const uint32_t g0 = 2u * (y0 * ncol + w);
    auto planes = [&](int k) -> Planes {
        const uint32_t g = g0 + 2u * (uint32_t)k * ncol + par(k);
        const uint4 q0 = philox_rk(g, a.sweep, 0u, tg_acc, a);
        const uint4 q1 = philox_rk(g, a.sweep, 1u, tg_acc, a);
        return Planes{{q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w}};
    };
    char* bits = reinterpret_cast<char*>(a.dst);
    auto at = [&](uint32_t off) -> uint32_t& { return *reinterpret_cast<uint32_t*>(bits + off); };
    Planes rnd[G::EARLY > 0 ? G::EARLY : 1];
#pragma unroll
    for (int k = 0; k < G::EARLY; ++k) rnd[k] = planes(k);
    grid_dep_launch();
    grid_dep_wait();
    // rows y0 - 1 .. y0 + T: the other colour's words (half 1 - p of a row
    // whose active half is p), and of rows y0 .. the active words and the edge
    // words: the even word to the right (p = 1), the odd word to the left (p = 0)
    const uint32_t c0 = y0 * pitch + 4 * w;  // the even word of row y0
    const uint32_t e1 = y0 * pitch + (w + 1 == ncol ? 0u : 4 * w + 4), e0 = y0 * pitch + half + (w == 0 ? half - 4 : 4 * w - 4);
    uint32_t g[T + 2], act[T], edge[T];
    g[0] = at((y0 == 0 ? c0 + (L - 1) * pitch : c0 - pitch) + (par(1) ? 0u : half));  // row y0 - 1 has row y0 + 1's parity
    g[T + 1] = at((y0 + T == L ? c0 - y0 * pitch : c0 + T * pitch) + (par(T) ? 0u : half));
#pragma unroll
    for (int k = 0; k < T; ++k) {
        const uint32_t p = par(k), rk = (uint32_t)k * pitch;
        g[k + 1] = at(c0 + rk + (p ? 0u : half));
        act[k] = at(c0 + rk + (p ? half : 0u));
        edge[k] = at((p ? e1 : e0) + rk);
    }
    int ntie = 0, esum = 0, msum = 0;
#pragma unroll
    for (int k = 0; k < T; ++k) {
        const uint32_t p = par(k);
        const uint32_t G1 = g[k + 1];
        const uint32_t Lb = p ? G1 : __funnelshift_l(edge[k], G1, 1);
        const uint32_t Rb = p ? __funnelshift_r(G1, edge[k], 1) : G1;
        uint32_t tie, inA;
        const Planes r = k < G::EARLY ? rnd[k < G::EARLY ? k : 0] : planes(k);
        const uint32_t An = decide_word(act[k], g[k], g[k + 2], Lb, Rb, r, th, tie, inA);
        const uint32_t off = c0 + (uint32_t)k * pitch + (p ? half : 0u);
        if (!live) tie = 0u;
        const uint32_t has = __ballot_sync(0xffffffffu, tie != 0u);
        if (tie) {
            const int e = ntie + __popc(has & ((1u << lane) - 1u));
            ties[warp][e] = make_uint4(off, tie, inA, An);
            tie_site[warp][e] = (y0 + (uint32_t)k) * L + 64u * w + p;
        }
        ntie += __popc(has);
        if (live) {
            at(off) = An;
            if (MEAS) {
                esum += word_bonds_unlike(An, g[k], g[k + 2], Lb, Rb);
                msum += 64 - 2 * __popc(An) - 2 * __popc(G1);
            }
        }
    }
    __syncwarp();
    for (int e = lane; e < ntie; e += 32) {
        const uint4 te = ties[warp][e];
        const uint32_t site = tie_site[warp][e];
        uint32_t flip = 0u;
        for (uint32_t m = te.y; m; m &= m - 1) {
            const int b = __ffs(m) - 1;
            const bool inA = (te.z >> b) & 1u;
            const uint64_t u53 = ((uint64_t)(inA ? a.tA8 : a.tB8) << 45) | (fine56_rk(site + 2u * (uint32_t)b, a) >> 11);
            if (u53 < (inA ? a.tA : a.tB)) {
                flip |= 1u << b;
                if (MEAS) {
                    // the tested classes have s * sum(nbrs) = +-2 (A) or +-4 (B) before the flip
                    esum += (inA ? 4 : 8) * (a.mode == 0 ? -1 : 1);
                    msum += (te.w >> b) & 1u ? 2 : -2;
                }
            }
        }
        // the word's only other writer in this launch stored it before the warp barrier
        if (flip) at(te.x) = te.w ^ flip;
    }
    if (MEAS) {
        esum = __reduce_add_sync(0xffffffffu, esum);
        msum = __reduce_add_sync(0xffffffffu, msum);
        if (lane == 0) {
            red[0][warp] = esum;
            red[1][warp] = msum;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            long long e = 0, m = 0;
            for (int k = 0; k < G::NT / 32; ++k) {
                e += red[0][k];
                m += red[1][k];
            }
            atomicAdd(reinterpret_cast<unsigned long long*>(a.acc + kAccEne), (unsigned long long)(2 * e));
            atomicAdd(reinterpret_cast<unsigned long long*>(a.acc + kAccMag), (unsigned long long)m);
        }
    }
}

// ---- layout conversion: row-major <-> split rows -----------------------------
// One thread moves a group of 64 consecutive sites of a row (x = 64w .. 64w+63):
// its even sites become word w of the even half, its odd sites word w of the
// odd half, each with the bytes transposed (split_addr): 16-byte loads and
// stores, byte moves in registers.

__device__ __forceinline__ void load64(const int8_t* __restrict__ p, uint8_t b[64])
{
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint4 v = reinterpret_cast<const uint4*>(p)[k];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 16; ++j) b[16 * k + j] = (uint8_t)(w[j >> 2] >> (8 * (j & 3)));
    }
}

__device__ __forceinline__ void load32(const int8_t* __restrict__ p, uint8_t b[32])
{
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint4 v = reinterpret_cast<const uint4*>(p)[k];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 16; ++j) b[16 * k + j] = (uint8_t)(w[j >> 2] >> (8 * (j & 3)));
    }
}

__device__ __forceinline__ void store32(int8_t* __restrict__ p, const uint8_t b[32])
{
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            w[j] = (uint32_t)b[16 * k + 4 * j] | ((uint32_t)b[16 * k + 4 * j + 1] << 8) |
                   ((uint32_t)b[16 * k + 4 * j + 2] << 16) | ((uint32_t)b[16 * k + 4 * j + 3] << 24);
        reinterpret_cast<uint4*>(p)[k] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

__global__ void split_rows(const int8_t* __restrict__ in, int8_t* __restrict__ out, int L)
{
    const int64_t groups = (int64_t)L * (L / 64);
    const int gpr = L / 64;
    for (int64_t gi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; gi < groups;
         gi += (int64_t)gridDim.x * blockDim.x) {
        const int64_t y = gi / gpr;
        const int w = (int)(gi - y * gpr);
        uint8_t b[64], e[32], o[32];
        load64(in + y * L + 64 * w, b);
#pragma unroll
        for (int s = 0; s < 32; ++s) {
            e[4 * (s & 7) + (s >> 3)] = b[2 * s];
            o[4 * (s & 7) + (s >> 3)] = b[2 * s + 1];
        }
        store32(out + y * L + 32 * w, e);
        store32(out + y * L + L / 2 + 32 * w, o);
    }
}

__global__ void merge_rows(const int8_t* __restrict__ in, int8_t* __restrict__ out, int L)
{
    const int64_t groups = (int64_t)L * (L / 64);
    const int gpr = L / 64;
    for (int64_t gi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; gi < groups;
         gi += (int64_t)gridDim.x * blockDim.x) {
        const int64_t y = gi / gpr;
        const int w = (int)(gi - y * gpr);
        uint8_t e[32], o[32], b[64];
        load32(in + y * L + 32 * w, e);
        load32(in + y * L + L / 2 + 32 * w, o);
#pragma unroll
        for (int s = 0; s < 32; ++s) {
            b[2 * s] = e[4 * (s & 7) + (s >> 3)];
            b[2 * s + 1] = o[4 * (s & 7) + (s >> 3)];
        }
        store32(out + y * L + 64 * w, b);
        store32(out + y * L + 64 * w + 32, b + 32);
    }
}

// Nonzero *flag when a byte of the row-major state is not a legal spin of
// the model (Ising: +-1; Potts: 0 .. q-1; Blume-Capel: -1, 0, 1).
__global__ void validate_int8(const int8_t* __restrict__ v, int64_t n, int kind, int q, int* __restrict__ flag)
{
    const int64_t n16 = n / 16;
    uint32_t bad = 0;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n16; k += (int64_t)gridDim.x * blockDim.x) {
        const uint4 x = reinterpret_cast<const uint4*>(v)[k];
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t ok;
            if (kind == MQV_MODEL_POTTS) ok = __vcmpltu4(w[j], 0x01010101u * (uint32_t)q);
            else if (kind == MQV_MODEL_BLUME_CAPEL) ok = __vcmpltu4(__vadd4(w[j], 0x01010101u), 0x03030303u);
            else ok = __vcmpeq4(w[j], 0x01010101u) | __vcmpeq4(w[j], 0xFFFFFFFFu);
            bad |= ~ok;
        }
    }
    for (int64_t i = 16 * n16 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int x = v[i];
        if (kind == MQV_MODEL_POTTS) bad |= (x < 0 || x >= q);
        else if (kind == MQV_MODEL_BLUME_CAPEL) bad |= (x < -1 || x > 1);
        else bad |= (x * x != 1);
    }
    if (__any_sync(0xffffffffu, bad != 0) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

// ---- host side ------------------------------------------------------------------

bool ising2d_supported(int L) { return L >= 64 && L % 64 == 0; }

typedef cudaError_t (*SweepLauncher)(const Ising2DArgs&, int, cudaStream_t);

template <int TX, int TY, int NWARP, bool MEAS>
static cudaError_t launch_t(const Ising2DArgs& a, int nsm, cudaStream_t stream)
{
    using G = TileGeom<TX, TY, NWARP>;
    auto kern = ising2d_sweep<TX, TY, NWARP, MEAS>;
    static std::atomic<int> cps{0};  // resident CTAs per SM for this instantiation (host threads share it)
    if (cps.load() == 0) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM);
        if (e != cudaSuccess) return e;
        int c = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, kern, NWARP * 32, G::SMEM);
        if (e != cudaSuccess) return e;
        cps = c < 1 ? 1 : c;
    }
    long long grid = (long long)nsm * cps;
    const long long need = (a.ntiles + NWARP - 1) / NWARP;
    if (grid > need) grid = need;
    kern<<<(int)grid, NWARP * 32, G::SMEM, stream>>>(a);
    return cudaGetLastError();
}

// RS / MINB: see ising2d_band; with MINB > 0 the grid has at most MINB CTAs
// per SM (longer bands re-read fewer halo rows).
template <int NT, int S, int NSB, bool MEAS, int W = 1, bool RS = false, int MINB = 0>
static cudaError_t launch_band(const Ising2DArgs& a, int nsm, cudaStream_t stream)
{
    using G = BandGeom<NT, S, NSB, W>;
    constexpr int SMEM = RS ? G::SMEM_RS : G::SMEM;
    auto kern = ising2d_band<NT, S, NSB, MEAS, W, RS, MINB>;
    static std::atomic<int> cps{0};  // resident CTAs per SM for this instantiation (host threads share it)
    if (cps.load() == 0) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return e;
        int c = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, kern, NT, SMEM);
        if (e != cudaSuccess) return e;
        if (MINB > 0 && c > MINB) c = MINB;
        cps = c < 1 ? 1 : c;
    }
    // one band per CTA, at least 8 rows each
    long long grid = (long long)nsm * cps;
    if (grid > G::L / 8) grid = G::L / 8;
    kern<<<(int)grid, NT, SMEM, stream>>>(a);
    return cudaGetLastError();
}

// Both colours of the colour kernel, in place on a.dst.
template <int T, bool MEAS>
static cudaError_t launch_colour(const Ising2DArgs& a, int, cudaStream_t stream)
{
    const unsigned nt = ColourGeom<T>::NT, grid = ((unsigned)(a.L >> 6) * (unsigned)(a.L / T) + nt - 1) / nt;
    const cudaError_t e = launch_pdl(ising2d_colour<T, false>, grid, nt, stream, a, 0);
    return e != cudaSuccess ? e : launch_pdl(ising2d_colour<T, MEAS>, grid, nt, stream, a, 1);
}

// Candidate kernels: tiles (tx x ty sites, nwarp independent warps per CTA)
// or bands (band = NT threads spanning a lattice of side 64 NT, ties resolved
// every S steps) or the colour kernel (T rows per thread).  Every candidate computes the same result; the autotuner
// keeps the fastest for a lattice size.
struct SweepConfig {
    int tx, ty, nwarp;  // tile shape (band: tx = L, ty = S, nwarp = NT / 32)
    bool band;
    int nsb;            // band: staged row slots
    SweepLauncher plain, meas;
    int w;              // band: word columns per thread
    int rs = 0;         // band: rows staged in registers, at most rs CTAs per SM (0: bulk-copy ring)
    int strip = 0;      // colour kernel: rows per thread (updates the state in place)
};

#define MQV_CFG(TX, TY, NW) \
    SweepConfig{TX, TY, NW, false, 0, launch_t<TX, TY, NW, false>, launch_t<TX, TY, NW, true>, 1}
#define MQV_BAND(NT, S, NSB) \
    SweepConfig{64 * NT, S, NT / 32, true, NSB, launch_band<NT, S, NSB, false>, launch_band<NT, S, NSB, true>, 1}
#define MQV_BANDW(NT, S, NSB, W)                                                                         \
    SweepConfig{64 * NT * W, S,                                                                          \
                NT / 32,     true,                                                                       \
                NSB,         launch_band<NT, S, NSB, false, W>,                                          \
                launch_band<NT, S, NSB, true, W>, W}

#define MQV_BANDRS(NT, S, W, MINB)                                                                        \
    SweepConfig{64 * NT * W, S, NT / 32, true, 0, launch_band<NT, S, 2, false, W, true, MINB>,             \
                launch_band<NT, S, 2, true, W, true, MINB>, W, MINB}

#define MQV_COLOUR(T) \
    SweepConfig{64, T, 1, false, 0, launch_colour<T, false>, launch_colour<T, true>, 1, 0, T}

static const SweepConfig kConfigs[] = {
    MQV_COLOUR(1), MQV_COLOUR(2), MQV_COLOUR(4),
    MQV_CFG(512, 32, 4), MQV_CFG(256, 32, 4), MQV_CFG(512, 32, 2), MQV_CFG(256, 32, 8),
    MQV_CFG(1024, 32, 2), MQV_CFG(128, 32, 4), MQV_CFG(64, 32, 4),
    MQV_BAND(256, 4, 2), MQV_BAND(256, 2, 2), MQV_BAND(256, 4, 3), MQV_BAND(256, 4, 4),
    MQV_BAND(128, 4, 2), MQV_BAND(128, 4, 4),
    MQV_BANDW(128, 4, 2, 2), MQV_BANDW(128, 2, 2, 2), MQV_BANDW(128, 1, 2, 2), MQV_BANDW(128, 3, 2, 2),
    MQV_BANDW(64, 4, 2, 2),
    MQV_BANDRS(128, 1, 2, 5), MQV_BANDRS(128, 1, 2, 6), MQV_BANDRS(128, 2, 2, 5),
    MQV_BANDRS(256, 1, 1, 3), MQV_BANDRS(256, 1, 1, 4),
    MQV_BANDRS(64, 2, 4, 4), MQV_BANDRS(64, 2, 4, 6), MQV_BANDRS(64, 2, 4, 8),
    MQV_BANDRS(64, 1, 4, 6), MQV_BANDRS(64, 1, 4, 8),
};
constexpr int kNumConfigs = (int)(sizeof(kConfigs) / sizeof(kConfigs[0]));

// Colour kernels up to here: at L = 8192 the 67 MB state still sits in the L2
// and two passes over it cost what the band kernel's single pass does (38.8
// against 41.4 us); at L = 16384 each pass goes to HBM (2 x 402 MB against 537).
// Below L = 2048 one row per thread is taken without timing (L = 1024: 7 us a
// sweep against 9 with four rows; tiles: 37.6 us).
constexpr int kColourMaxLen = 8192;
static bool config_fits(const SweepConfig& c, int L)
{
    if (c.band) return L == c.tx;
    if (c.strip) return L <= kColourMaxLen;
    return L % c.tx == 0 && L % c.ty == 0;
}

static void fill_args(Sim* s, const SweepConfig& c, long long* acc, Ising2DArgs& a)
{
    a.src = (const int8_t*)s->state[s->cur];
    a.dst = (int8_t*)s->state[c.strip ? s->cur : s->cur ^ 1];
    a.L = s->len;
    a.ntx = c.band ? 1 : s->len / c.tx;
    a.ntiles = c.band ? 0 : a.ntx * (s->len / c.ty);
    a.key = make_key(s->seed);
    for (int r = 0; r < 10; ++r) {
        a.rk0[r] = a.key.k0 + (uint32_t)r * 0x9E3779B9u;
        a.rk1[r] = a.key.k1 + (uint32_t)r * 0xBB67AE85u;
    }
    a.sweep = (uint32_t)s->sweep;
    a.replica = s->replica;
    // cuts of update_accepted<1> on u53 per aligned-neighbour count k:
    // dE = J (s_new - s_old) sum_nbrs = J (8 - 4k)
    if (s->thr_J != s->md.J || s->thr_beta != s->md.beta) {
        for (int k = 0; k < 5; ++k) s->thr_cut[k] = accept_cut(1, s->md.J * (double)(8 - 4 * k), s->md.beta);
        s->thr_J = s->md.J;
        s->thr_beta = s->md.beta;
    }
    // the tested classes: aligned counts 3 and 4 for J < 0, 1 and 0 for J > 0
    const double J = s->md.J;
    const int ka = J < 0 ? 3 : 1, kb = J < 0 ? 4 : 0;
    a.mode = J < 0 ? 0 : (J > 0 ? 1 : 2);
    const unsigned long long TA = s->thr_cut[ka], TB = s->thr_cut[kb];
    a.useA = TA < (1ull << 53);
    a.useB = TB < (1ull << 53);
    a.tA = TA;
    a.tB = TB;
    a.tA8 = (uint32_t)(TA >> 45) & 0xFFu;
    a.tB8 = (uint32_t)(TB >> 45) & 0xFFu;
    a.acc = acc;
    a.status = s->d_status;
    a.counter = s->d_counter;
    a.wait_ns = 2000000000ull;  // 2 s
    a.withhold = -1;
}

// Time every fitting candidate on this lattice (sweeps into the scratch
// buffer; the state is not modified) and keep the fastest.  Small
// lattices take the first fitting candidate.
static void config_name(const SweepConfig& c, char* buf, int len)
{
    if (c.strip) snprintf(buf, len, "ising2d_colour<%d>", c.strip);
    else if (c.band && c.rs) snprintf(buf, len, "ising2d_band_rs<%d,%d,%d,%d>", c.nwarp * 32, c.ty, c.w, c.rs);
    else if (c.band && c.w > 1) snprintf(buf, len, "ising2d_band<%d,%d,%d,%d>", c.nwarp * 32, c.ty, c.nsb, c.w);
    else if (c.band) snprintf(buf, len, "ising2d_band<%d,%d,%d>", c.nwarp * 32, c.ty, c.nsb);
    else snprintf(buf, len, "ising2d_sweep<%d,%d,%d>", c.tx, c.ty, c.nwarp);
}

static int pick_config(Sim* s)
{
    // MARQOV_B200_SWEEP_CONFIG=<name> (as mqv_describe prints it) forces one
    // candidate, when it fits the lattice: for tests of each kernel shape
    if (const char* want = getenv("MARQOV_B200_SWEEP_CONFIG")) {
        char buf[64];
        for (int k = 0; k < kNumConfigs; ++k) {
            config_name(kConfigs[k], buf, sizeof buf);
            if (config_fits(kConfigs[k], s->len) && strcmp(buf, want) == 0) return k;
        }
    }
    int first = -1;
    for (int k = 0; k < kNumConfigs; ++k)
        if (config_fits(kConfigs[k], s->len)) {
            first = k;
            break;
        }
    if (s->len < 2048 || first < 0) return first;
    cudaEvent_t e0, e1;
    if (cudaEventCreate(&e0) != cudaSuccess) return first;
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return first;
    }
    // two rounds over the candidates, four timed sweeps each, the best of
    // the rounds per candidate: a candidate timed while the clocks still
    // ramp up gets a second chance
    int best = first;
    float best_ms = 1e30f;
    constexpr int kRounds = 2, kTimed = 4;
    for (int round = 0; round < kRounds; ++round)
        for (int k = 0; k < kNumConfigs; ++k) {
            if (!config_fits(kConfigs[k], s->len)) continue;
            // tiles are never the fastest where the colour kernels apply
            // (L = 2048: 37 against 12 us, L = 4096: 51 against 12 us)
            if (s->len <= kColourMaxLen && !kConfigs[k].band && !kConfigs[k].strip) continue;
            Ising2DArgs a{};
            fill_args(s, kConfigs[k], nullptr, a);
            a.dst = (int8_t*)s->state[s->cur ^ 1];  // in-place kernels too: the state stays as it is
            cudaMemsetAsync(s->d_counter, 0, sizeof(int), s->stream);
            if (kConfigs[k].plain(a, s->num_sms, s->stream) != cudaSuccess) continue;  // warm-up
            cudaEventRecord(e0, s->stream);
            for (int i = 0; i < kTimed; ++i) {
                cudaMemsetAsync(s->d_counter, 0, sizeof(int), s->stream);
                kConfigs[k].plain(a, s->num_sms, s->stream);
            }
            cudaEventRecord(e1, s->stream);
            s->launches += 1 + kTimed;
            float ms = 0;
            if (cudaEventSynchronize(e1) == cudaSuccess && cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess &&
                ms < best_ms) {
                best_ms = ms;
                best = k;
            }
        }
    cudaGetLastError();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return best;
}

// A band configuration with the bulk-copy ring (and its bounded waits) that
// fits the lattice (-1: none), for the injected timeout.
int ising2d_band_config(const Sim* s)
{
    for (int k = 0; k < kNumConfigs; ++k)
        if (kConfigs[k].band && !kConfigs[k].rs && config_fits(kConfigs[k], s->len)) return k;
    return -1;
}

// ---- host side of the bit planes ---------------------------------------------------

template <int T>
static cudaError_t launch_bits_t(const Ising2DArgs& a, cudaStream_t stream)
{
    const unsigned nt = BitsGeom<T>::NT, grid = ((unsigned)(a.L >> 6) * (unsigned)(a.L / T) + nt - 1) / nt;
    const cudaError_t e = launch_pdl(ising2d_bits<T, 0, false>, grid, nt, stream, a);
    if (e != cudaSuccess) return e;
    return a.acc ? launch_pdl(ising2d_bits<T, 1, true>, grid, nt, stream, a)
                 : launch_pdl(ising2d_bits<T, 1, false>, grid, nt, stream, a);
}

// Rows per thread: one shortens a launch, more share the neighbour rows and the
// set-up (us per sweep with 1 / 2 / 4 / 8 rows: L = 1024 4.3 / 4.4 / 5.9 / 7.8, L =
// 4096 9.3 / 7.7 / 9.8 / 12, L = 8192 31 / 24.5 / 21.2 / 22.3, L = 16384 118 / 92 / 77
// / 71).
static int bits_rows(int L) { return L < 3072 ? 1 : L < 6144 ? 2 : L < 12288 ? 4 : 8; }
// Sweeps in a row from which packing and unpacking pay (us, int8 and bits: 3
// sweeps at L = 16384 340 and 318, at L = 4096 38 and 36; 2 at L = 16384 227 and
// 247, at L = 4096 26 and 28; at L = 1024 3 sweeps 17 and 18, 20 sweeps 115 and 87).
static int bits_min_sweeps(int L) { return L < 2048 ? 5 : 3; }

static void bits_name(const Sim* s, char* buf, int len) { snprintf(buf, len, "ising2d_bits<%d>", s->bits_rows); }

// whether `sweeps` sweeps in a row run on bit planes
bool ising2d_use_bits(Sim* s, int64_t sweeps)
{
    if (!s->fused_ising2d || s->inject_row >= 0) return false;
    if (s->bits_rows < 0) {
        // MARQOV_B200_SWEEP_CONFIG: ising2d_bits<T> takes the bit planes for any
        // number of sweeps, another kernel's name never
        s->bits_rows = bits_rows(s->len);
        s->bits_min = bits_min_sweeps(s->len);
        if (const char* want = getenv("MARQOV_B200_SWEEP_CONFIG")) {
            int t = 0;
            const bool named = sscanf(want, "ising2d_bits<%d>", &t) == 1 && (t == 1 || t == 2 || t == 4 || t == 8);
            if (named) s->bits_rows = t;
            s->bits_min = named ? 1 : 0;
        }
    }
    return s->bits_min > 0 && sweeps >= s->bits_min;
}

// The state to bit planes in the spare buffer; until ising2d_bits_end the
// sweeps (launch_ising2d_sweep) run there.
cudaError_t ising2d_bits_begin(Sim* s)
{
    const int64_t words = s->n / 32;
    ising2d_pack<<<(unsigned)((words + 255) / 256), 256, 0, s->stream>>>((const int8_t*)s->state[s->cur],
                                                                        (uint32_t*)s->state[s->cur ^ 1], words);
    s->launches++;
    s->bits_on = true;
    return cudaGetLastError();
}

cudaError_t ising2d_bits_end(Sim* s)
{
    const int64_t words = s->n / 32;
    s->launches++;
    s->bits_on = false;
    s->bits_last = true;
    return launch_pdl(ising2d_unpack, (unsigned)((words + 255) / 256), 256, s->stream,
                      (const uint32_t*)s->state[s->cur ^ 1], (int8_t*)s->state[s->cur], words);
}

static cudaError_t launch_bits_sweep(Sim* s, long long* acc)
{
    Ising2DArgs a{};
    fill_args(s, kConfigs[0], acc, a);
    a.dst = (int8_t*)s->state[s->cur ^ 1];
    s->launches += 2;
    switch (s->bits_rows) {
        case 1: return launch_bits_t<1>(a, s->stream);
        case 2: return launch_bits_t<2>(a, s->stream);
        case 4: return launch_bits_t<4>(a, s->stream);
        default: return launch_bits_t<8>(a, s->stream);
    }
}

cudaError_t launch_ising2d_sweep(Sim* s, long long* acc)
{
    if (s->bits_on) return launch_bits_sweep(s, acc);
    s->bits_last = false;
    if (s->inject_row >= 0) s->sweep_cfg = ising2d_band_config(s);
    if (s->sweep_cfg < 0) {
        s->sweep_cfg = pick_config(s);
        if (s->sweep_cfg < 0) return cudaErrorInvalidValue;
    }
    const SweepConfig& c = kConfigs[s->sweep_cfg];
    Ising2DArgs a{};
    fill_args(s, c, acc, a);
    if (s->inject_row >= 0) {  // one sweep only
        a.withhold = s->inject_row;
        a.wait_ns = s->inject_wait_ns;
        s->inject_row = -1;
    }
    if (!c.band && !c.strip) {  // tiles are taken from a counter; bands are fixed per CTA
        const cudaError_t e = cudaMemsetAsync(s->d_counter, 0, sizeof(int), s->stream);
        if (e != cudaSuccess) return e;
    }
    const cudaError_t e = acc ? c.meas(a, s->num_sms, s->stream) : c.plain(a, s->num_sms, s->stream);
    s->launches += c.strip ? 2 : 1;
    if (!c.strip) s->cur ^= 1;
    return e;
}

const char* ising2d_config_name(Sim* s, char* buf, int len)
{
    if (s->bits_last) {
        bits_name(s, buf, len);
        return buf;
    }
    if (s->sweep_cfg < 0) return "";
    config_name(kConfigs[s->sweep_cfg], buf, len);
    return buf;
}

cudaError_t launch_split_rows(Sim* s, const void* rowmajor, void* split)
{
    split_rows<<<148 * 8, 256, 0, s->stream>>>((const int8_t*)rowmajor, (int8_t*)split, s->len);
    s->launches++;
    return cudaGetLastError();
}

cudaError_t launch_merge_rows(Sim* s, const void* split, void* rowmajor)
{
    merge_rows<<<148 * 8, 256, 0, s->stream>>>((const int8_t*)split, (int8_t*)rowmajor, s->len);
    s->launches++;
    return cudaGetLastError();
}

cudaError_t launch_validate_int8(Sim* s, const void* rowmajor, int* flag)
{
    validate_int8<<<148 * 8, 256, 0, s->stream>>>((const int8_t*)rowmajor, s->n, s->md.kind, s->md.q, flag);
    s->launches++;
    return cudaGetLastError();
}

}  // namespace mqv
