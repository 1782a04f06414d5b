// EMCS without clusters of Ising-type models on CSR graphs (Ising, embedded
// Ising, Edwards-Anderson with any bonds) in one launch per chunk, on a
// thread-block cluster, for sm_100a.
//
// A greedily coloured graph has a dozen or more colours, most of them small,
// and a launch per colour costs more than its work (a random geometric graph
// of 131,072 sites: 14 launches of 5 us a sweep, 6.8 us apart on the host).
// Here one cluster of up to 16 CTAs runs whole chunks of sweeps and
// measurements, the colours in turn.  Every CTA keeps the spins of the whole
// graph as bits in its shared memory, so that a site gathers its neighbours
// there.  The bits lie in the order of (CTA, colour): a warp updates the 32
// sites of one word, and sends the word to every CTA (st.async, 4 bytes to
// each from a lane of its own; its own CTA too).  A warp begins the next colour
// when all words of this one have arrived, counted by an mbarrier -- which
// also tells that every other warp has read what is about to change -- so a
// colour needs no cluster barrier.
// The initial state is step 0, the colours are steps 1, 2, ...; the words of
// even steps count at one mbarrier, those of odd steps at the other.  Two rules
// make that enough:
//   * every CTA sends at least one word of every step (colours without a site
//     are left out, a CTA without a site of a colour has a word of padding).
//     So no word of step t + 2 is sent before step t has ended everywhere:
//     its sender has the words of step t + 1 of every CTA, each sent after
//     step t had ended there;
//   * a CTA barrier comes before every wait.  Thread 0 arms step t + 1 behind
//     it, so no barrier runs past a thread that still waits for step t - 1, and
//     no thread waits for step t before thread 0 has armed it: the parity of
//     the wait is unambiguous.
// Waits are bounded.  A thread whose wait ran out sets the error status and
// waits, sends and arms no more; its CTA learns of it before the next sweep or
// measurement and skips the rest of the run, the other threads and CTAs run out in
// turn for want of its words.  Every
// CTA passes the same cluster barriers whether it runs or skips, and one that
// gave up stays a while after the last of them, since words of others may still
// be on their way to it.
// What does not depend on the spins,
// a site and its neighbours' bits, is fetched ahead.  The neighbour lists lie
// in slices of 32 positions, one row per neighbour, so that a warp reads them
// in whole lines; a sweep's acceptance planes are drawn once per CTA for the
// range of sites that it owns.  Same words, decisions and order of colours as
// metro_int8_csr, same sums as measure_int8.  Bound by the latency of a
// colour (gather, decision, words on their way).  Per sweep, launches and
// this kernel (us): 1000 sites 45 and 9.4, 16,384 sites 72 and 12.2, 131,072 sites
// 92 and 47, 262,144 sites 101 and 85.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <vector>

#include "int8_site.cuh"

namespace cg = cooperative_groups;

namespace mqv {

constexpr int kEllThreads = 512;
constexpr int kEllMaxCtas = 16;
constexpr int kEllRounds = 2048;        // rounds of a sweep
constexpr int kEllNb = 16;  // neighbours held ahead per site; further ones are read after the barrier
constexpr size_t kEllMaxSmem = 224 * 1024;

// 4 bytes to a CTA's shared memory, counted by an mbarrier there
__device__ __forceinline__ void st_async(uint32_t dst, uint32_t v, uint32_t bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(v), "r"(bar)
                 : "memory");
}
// address of a shared-memory location of this CTA in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// shared memory: the sweep's rounds, the graph's spins (a bit per position,
// set: -1), the acceptance planes of one CTA's range (run, parity, half)
static size_t ell_smem(size_t npos, int range, int rounds)
{
    return (((size_t)rounds * 16 + npos / 8 + 15) & ~(size_t)15) + (size_t)range;
}

// a position of a CTA's colour order and what is known of it before its colour
struct EllPos {
    int site, deg;  // site -1: none
    int64_t nb;     // its slice's neighbours in EllDev::nb
};

struct EllRun {
    EllDev g;
    int64_t n;
    int8_t* s;
    Key key;
    uint32_t sweep0, replica;
    int n_emcs, nmetro, D;  // D: middle of the cut table
    const unsigned long long* cuts;
    long long* acc;  // measurement accumulators of the first EMCS, or NULL
    int* status;     // device error word
    unsigned long long wait_ns;
    int hold;        // the colour of the run (from 1) of which CTA 0 withholds a word (tests); 0: none
};

template <bool BONDS>
__global__ void __launch_bounds__(kEllThreads, 1) ell_emcs(EllRun R)
{
    extern __shared__ __align__(16) unsigned char smem[];
    cg::cluster_group cl = cg::this_cluster();
    const int me = (int)cl.block_rank(), ctas = (int)cl.num_blocks();
    const EllDev& g = R.g;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // A sweep is a sequence of rounds of at most kEllThreads positions of one
    // colour: first position, one past the last, whether the colour begins
    // (then the bytes of its words over all CTAs).
    int4* rounds = reinterpret_cast<int4*>(smem);
    uint32_t* bits = reinterpret_cast<uint32_t*>(rounds + g.rounds);
    uint4* tab = reinterpret_cast<uint4*>(smem + (((size_t)g.rounds * 16 + (size_t)g.npos / 8 + 15) & ~(size_t)15));
    __shared__ int s_rounds;
    // words of even and of odd steps (one of step t + 1 may come before the last
    // of step t)
    __shared__ __align__(8) uint64_t bars[2];
    const int lo = me * g.range;  // this CTA's sites [lo, lo + range)
    const int32_t* cptr = g.cptr + me * g.ncol;
    const int p0 = cptr[0], p1 = cptr[g.ncol];
    if (tid == 0) {
        int r = 0;
        for (int c = 0; c < g.ncol; ++c) {
            const int end = cptr[c + 1];
            for (int p = cptr[c]; p < end; p += kEllThreads)
                rounds[r++] = make_int4(p, min(p + kEllThreads, end), p == cptr[c], g.cwords[c] * 4);
        }
        s_rounds = r;
        mbar_init(smem_addr(&bars[0]), 1);
        mbar_init(smem_addr(&bars[1]), 1);
        mbar_fence_init();
    }
    cl.sync();  // every CTA runs, its barriers are set up
    const int nround = s_rounds;
    // lane q sends the warp's words to CTA q
    const bool sends = lane < ctas;
    const uint32_t to = sends ? map_rank(smem_addr(bits), (uint32_t)lane) : 0u;
    const uint32_t to_bar = sends ? map_rank(smem_addr(&bars[0]), (uint32_t)lane) : 0u;
    int step = 0;       // steps begun
    bool stop = false;  // a wait of this thread ran out
    bool over = false;  // ... of this CTA, as of the last meet()
    auto meet = [&]() { stop = over = __syncthreads_or(stop); };
    auto arm = [&](int bytes) {
        if (tid == 0 && !stop) mbar_expect_tx(smem_addr(&bars[step & 1]), (uint32_t)bytes);
        ++step;
    };
    const int hold = R.hold && me == 0 && warp == 0 ? R.hold + 1 : 0;  // the step of the withheld word
    auto send = [&](int word, uint32_t v) {
        if (sends && !stop) st_async(to + 4u * (uint32_t)word, v, to_bar + 8u * (uint32_t)((step - 1) & 1));
    };
    // until every word of the last step begun has arrived, behind a CTA barrier
    // (bounded: a lost word sets the error status and ends the run).  The wait
    // acquires at CTA scope: what it guards lies in this CTA's shared memory, where
    // a word lands before it is counted.  At cluster scope it drops the L1, and
    // with it the neighbour lists, at every colour (16,384 sites 12.2 -> 15.6 us a
    // sweep).
    auto receive = [&]() {
        if (stop) return;
        const uint32_t bar = smem_addr(&bars[(step - 1) & 1]), par = (uint32_t)((step - 1) >> 1) & 1u;
        if (mbar_try_wait(bar, par)) return;
        const uint64_t t0 = global_timer_ns();
        for (uint32_t k = 1; !mbar_try_wait(bar, par); ++k)
            if ((k & 255u) == 0 && global_timer_ns() - t0 > R.wait_ns) {
                stop = true;
                atomicExch(R.status, MQV_ERR_TIMEOUT);
                break;
            }
    };
    arm(g.npos / 8);
    for (int p = p0 + warp * 32; p < p1; p += 4 * kEllThreads) {
        int8_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int q = p + k * kEllThreads + lane, i = q < p1 ? g.site[q] : -1;
            v[k] = i >= 0 ? R.s[i] : (int8_t)1;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t m = __ballot_sync(0xffffffffu, v[k] < 0);
            if (p + k * kEllThreads < p1) send((p + k * kEllThreads) >> 5, m);
        }
    }
    auto find = [&](int p, int end) -> EllPos {
        EllPos q{-1, 0, 0};
        if (p < end) {
            q.site = g.site[p];
            q.deg = g.deg[p];
            q.nb = g.slice[p >> 5];
        }
        return q;
    };
    auto find_round = [&](int r) -> EllPos {
        const int4 rd = rounds[r];
        return find(rd.x + tid, rd.y);
    };
    auto minus = [&](int j) -> int { return (int)((bits[j >> 5] >> (j & 31)) & 1u); };
    struct Pre {
        int nbr[kEllNb], w[kEllNb];
    };
    auto fetch = [&](const EllPos& q) -> Pre {
        Pre e;
        const int32_t* nb = g.nb + q.nb + lane;
        const int8_t* bd = BONDS ? g.bonds + q.nb + lane : nullptr;
#pragma unroll
        for (int t = 0; t < kEllNb; ++t) {
            e.nbr[t] = t < q.deg ? nb[32 * t] : -1;
            e.w[t] = BONDS && t < q.deg ? (int)bd[32 * t] : 1;
        }
        return e;
    };
    // sum over the neighbours of their spins (bond weights)
    auto field = [&](const EllPos& q, const Pre& e) -> int {
        int sum = BONDS ? 0 : q.deg;
#pragma unroll
        for (int t = 0; t < kEllNb; ++t)
            if (e.nbr[t] >= 0) sum += BONDS ? e.w[t] * (1 - 2 * minus(e.nbr[t])) : -2 * minus(e.nbr[t]);
        for (int t = kEllNb; t < q.deg; ++t) {
            const int j = g.nb[q.nb + lane + 32 * t];
            sum += BONDS ? (int)g.bonds[q.nb + lane + 32 * t] * (1 - 2 * minus(j)) : -2 * minus(j);
        }
        return sum;
    };
    const uint32_t c3a = tag(kAccept, R.replica);
    // the next round's site, and the round's after it, fetched ahead
    EllPos cur = find_round(0);
    int ahead = nround > 1 ? 1 : 0;  // the round of `next`
    EllPos next = find_round(ahead);
    Pre pre = fetch(cur);
    for (int em = 0; em < R.n_emcs; ++em) {
        for (int j = 0; j < R.nmetro && !over; ++j) {
            const uint32_t sweep = R.sweep0 + (uint32_t)(em * R.nmetro + j);
            // the sweep's acceptance planes of this CTA's sites
            meet();
            if (over) break;
            for (int q = tid; q < g.range / 16; q += kEllThreads)
                tab[q] = philox(((uint32_t)(lo >> 6) + ((uint32_t)q >> 2)) * 2u + (((uint32_t)q >> 1) & 1u), sweep,
                                (uint32_t)q & 1u, c3a, R.key);
            for (int r = 0; r < nround; ++r) {
                const EllPos q = cur;
                const Pre e = pre;
                ahead = ahead + 1 == nround ? 0 : ahead + 1;
                cur = next;
                pre = fetch(cur);
                next = find_round(ahead);
                const int4 rd = rounds[r];
                if (rd.z) {  // a colour begins
                    __syncthreads();  // also: the sweep's planes are there
                    receive();
                    arm(rd.w);
                }
                bool flip = false;
                if (q.site >= 0) {
                    const int old = 1 - 2 * minus(rd.x + tid);
                    const unsigned long long cut = R.cuts[old * field(q, e) + R.D];
                    flip = accept_top_or_fine(cut, accept_top8_tab(tab, (uint32_t)lo >> 6, (uint32_t)q.site), R.key,
                                              (uint32_t)q.site, sweep, R.replica);
                }
                const uint32_t m = __ballot_sync(0xffffffffu, flip);
                const int word = (rd.x + warp * 32) >> 5;
                if (rd.x + warp * 32 < rd.y && step != hold) send(word, bits[word] ^ m);
            }
        }
        if (!R.acc) continue;
        // measurement: the field of every site of this CTA, all colours
        meet();
        if (!over) receive();
        long long ene = 0;
        int down = 0, p = over ? p1 : p0 + tid;
        EllPos q = find(p, p1), q2 = find(p + kEllThreads, p1);
        Pre e = fetch(q);
        for (; p < p1; p += kEllThreads) {
            const EllPos q3 = find(p + 2 * kEllThreads, p1);
            const Pre e2 = fetch(q2);
            if (q.site >= 0) {
                const int dn = minus(p);
                ene += (1 - 2 * dn) * field(q, e);
                down += dn;
            }
            q = q2;
            e = e2;
            q2 = q3;
        }
        ene = warp_sum_ll(ene);
        down = __reduce_add_sync(0xffffffffu, down);
        if (lane == 0) {
            unsigned long long* a = reinterpret_cast<unsigned long long*>(R.acc + (int64_t)em * kAccStride);
            atomicAdd(a + kAccEne, (unsigned long long)ene);
            atomicAdd(a + kAccMag, (unsigned long long)(-2ll * down));
            if (me == 0 && warp == 0) {
                atomicAdd(a + kAccMag, (unsigned long long)R.n);
                atomicAdd(a + kAccSq, (unsigned long long)R.n);
            }
        }
        cl.sync();  // the next sweep's words would arrive while others still read
    }
    meet();
    if (!over) {
        receive();
        for (int p = p0 + tid; p < p1; p += kEllThreads) {
            const int i = g.site[p];
            if (i >= 0) R.s[i] = (int8_t)(1 - 2 * minus(p));
        }
    }
    cl.sync();  // no CTA leaves while words are on their way to it or from it
    if (stop) {
        // the last words sent are older than the barrier: 20 us are enough for them
        const uint64_t t0 = global_timer_ns();
        for (int k = 0; k < 1 << 16 && global_timer_ns() - t0 < 20000; ++k) __nanosleep(200);
    }
}

typedef void (*EllKernel)(EllRun);
static EllKernel ell_kernel(bool bonds) { return bonds ? ell_emcs<true> : ell_emcs<false>; }

static void ell_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int ctas, size_t smem, cudaStream_t st)
{
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kEllThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}

// Largest cluster of up to 16 CTAs the device runs (sizes above 8 are not
// portable), asked once per device; sets the kernels' attributes.
static int ell_max_ctas(int device)
{
    static std::atomic<int> known[64] = {};  // host threads share it
    if (device >= 0 && device < 64 && known[device]) return known[device];
    int best = 1;
    for (bool b : {false, true}) {
        cudaFuncSetAttribute(ell_kernel(b), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEllMaxSmem);
        cudaFuncSetAttribute(ell_kernel(b), cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    for (int c = kEllMaxCtas; c > 1 && best == 1; c /= 2) {
        cudaLaunchAttribute at[1];
        cudaLaunchConfig_t cfg;
        ell_config(cfg, at, c, kEllMaxSmem, nullptr);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, ell_kernel(true), &cfg) == cudaSuccess && n > 0) best = c;
    }
    cudaGetLastError();
    if (device >= 0 && device < 64) known[device] = best;
    return best;
}

// Positions of a coloured graph on `ctas` CTAs of `range` sites: the site of
// every position (-1: padding), the positions of every (CTA, colour), at least
// one word each, and the words of every colour.  Colours without a site are
// left out, the others keep their order.
struct EllLayout {
    int ncol = 0;
    std::vector<int32_t> site, cptr, cwords;
};
static int64_t ell_range(int64_t n, int ctas) { return ((n + ctas - 1) / ctas + 63) / 64 * 64; }
static EllLayout ell_layout(int64_t n, const int32_t* col, int ctas)
{
    EllLayout e;
    const int64_t range = ell_range(n, ctas);
    std::vector<int32_t> used;  // colour -> its place among those that have sites
    for (int64_t i = 0; i < n; ++i) {
        if ((size_t)col[i] >= used.size()) used.resize((size_t)col[i] + 1, 0);
        used[(size_t)col[i]] = 1;
    }
    for (int32_t& u : used) u = u ? e.ncol++ : -1;
    e.cptr.assign((size_t)ctas * e.ncol + 1, 0);
    e.cwords.assign((size_t)e.ncol, 0);
    e.site.reserve((size_t)n + (size_t)ctas * e.ncol * 32);
    std::vector<std::vector<int32_t>> bins((size_t)e.ncol);
    for (int r = 0; r < ctas; ++r) {
        for (auto& b : bins) b.clear();
        for (int64_t i = r * range; i < std::min(n, (r + 1) * range); ++i)
            bins[(size_t)used[(size_t)col[i]]].push_back((int32_t)i);
        for (int c = 0; c < e.ncol; ++c) {
            const size_t first = e.site.size();
            e.site.insert(e.site.end(), bins[(size_t)c].begin(), bins[(size_t)c].end());
            while (e.site.size() == first || e.site.size() % 32) e.site.push_back(-1);  // a colour starts a slice
            e.cptr[(size_t)r * e.ncol + c + 1] = (int32_t)e.site.size();
            e.cwords[(size_t)c] += (int32_t)((e.site.size() - first) / 32);
        }
    }
    return e;
}

// The sliced neighbour lists of a coloured graph (col: every site's colour),
// built on the host and uploaded; nothing where the graph does not fit.
cudaError_t build_ell(Sim* s, int64_t n, const int32_t* rp, const int32_t* ci, const int8_t* bonds,
                      const std::vector<int32_t>& col)
{
    const int most = ell_max_ctas(s->device);
    int ncol = 0;  // colours that have sites
    for (size_t c = 0; c + 1 < s->colour_ptr.size(); ++c) ncol += s->colour_ptr[c + 1] > s->colour_ptr[c];
    // a CTA per 1024 sites (us per sweep with one per 1024 / 4096 / 8192: 4096
    // sites 12 / 17 / 17, 16,384 sites 12 / 22 / 31)
    int ctas = 1;
    while (ctas < most && n > (int64_t)ctas * 1024) ctas *= 2;
    const int64_t range64 = ell_range(n, ctas);
    const int64_t most_rounds = ncol + (range64 + 32 * (int64_t)ncol) / kEllThreads + 1;  // colours are padded to 32
    const int64_t most_pos = n + 32 * (int64_t)ncol * ctas;
    if (most_pos >= (int64_t)1 << 31 || range64 * ctas >= (int64_t)1 << 31 || most_rounds > kEllRounds ||
        ell_smem((size_t)most_pos, (int)range64, (int)most_rounds) > kEllMaxSmem)
        return cudaSuccess;
    const int range = (int)range64;
    const EllLayout lay = ell_layout(n, col.data(), ctas);
    const std::vector<int32_t>&site = lay.site, &cptr = lay.cptr, &cwords = lay.cwords;
    std::vector<int32_t> deg;
    const size_t np = site.size();
    // bytes of a step's words count at one mbarrier: at most 2^20 - 1
    std::vector<int32_t> pos((size_t)n, 0);
    if (np / 8 >= (size_t)1 << 20) return cudaSuccess;
    for (size_t p = 0; p < np; ++p)
        if (site[p] >= 0) pos[(size_t)site[p]] = (int32_t)p;
    deg.resize(np);
    for (size_t p = 0; p < np; ++p) deg[p] = site[p] < 0 ? 0 : rp[site[p] + 1] - rp[site[p]];
    std::vector<int64_t> slice;
    int64_t total = 0;
    for (size_t p = 0; p < np; p += 32) {
        slice.push_back(total);
        total += 32 * (int64_t)*std::max_element(deg.begin() + (int64_t)p, deg.begin() + (int64_t)p + 32);
    }
    // few large degrees among small ones of their colour: the slices would take
    // many times the graph's memory, the launches take none
    if (total > std::min<int64_t>(8 * (int64_t)rp[n] + (1 << 20), (int64_t)1 << 29)) return cudaSuccess;
    std::vector<int32_t> nb((size_t)std::max<int64_t>(total, 1), 0);
    std::vector<int8_t> bd(bonds ? nb.size() : 0, 0);
    for (size_t p = 0; p < np; ++p)
        for (int t = 0; t < deg[p]; ++t) {
            const size_t at = (size_t)slice[p >> 5] + (p & 31) + 32 * (size_t)t;
            nb[at] = pos[(size_t)ci[rp[site[p]] + t]];
            if (bonds) bd[at] = bonds[rp[site[p]] + t];
        }
    // one allocation: slices, then 4-byte tables, then bonds
    const size_t bytes = slice.size() * 8 + (cptr.size() + cwords.size() + 2 * np + nb.size()) * 4 + bd.size();
    char* d = nullptr;
    cudaError_t e = cudaMalloc(&d, bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return cudaSuccess;  // the launch-per-colour path needs no tables
    }
    s->d_ell = d;
    size_t off = 0;
    auto put = [&](const void* src, size_t size) -> const void* {
        const char* at = d + off;
        off += size;
        if (e == cudaSuccess) e = upload_sync(s->stream, (void*)at, src, size);
        return at;
    };
    s->ell.slice = (const int64_t*)put(slice.data(), slice.size() * 8);
    s->ell.cptr = (const int32_t*)put(cptr.data(), cptr.size() * 4);
    s->ell.cwords = (const int32_t*)put(cwords.data(), cwords.size() * 4);
    s->ell.site = (const int32_t*)put(site.data(), np * 4);
    s->ell.deg = (const int32_t*)put(deg.data(), np * 4);
    s->ell.nb = (const int32_t*)put(nb.data(), nb.size() * 4);
    s->ell.bonds = bonds ? (const int8_t*)put(bd.data(), bd.size()) : nullptr;
    s->ell.ncol = ncol;
    s->ell.ctas = ctas;
    s->ell.range = range;
    s->ell.rounds = (int)most_rounds;
    s->ell.npos = (int)np;
    return e;
}

// The words of every colour and CTA (colour by colour) of such a layout, as far
// as `room` goes; returns the colours that have sites.
int ell_words(int64_t n, const int32_t* col, int ctas, int32_t* words, int64_t room)
{
    const EllLayout e = ell_layout(n, col, ctas);
    for (int c = 0; c < e.ncol; ++c)
        for (int r = 0; r < ctas; ++r) {
            const size_t k = (size_t)r * e.ncol + c;
            if ((int64_t)c * ctas + r < room) words[(size_t)c * ctas + r] = (e.cptr[k + 1] - e.cptr[k]) / 32;
        }
    return e.ncol;
}

cudaError_t ensure_cuts(Sim* s);

// n_emcs times nmetro sweeps (and a measurement into acc slots 0 .. when acc is
// given) of a graph in one launch; advances the counter.
cudaError_t launch_ell_emcs(Sim* s, int n_emcs, int nmetro, long long* acc)
{
    cudaError_t e = ensure_cuts(s);
    if (e != cudaSuccess) return e;
    ell_max_ctas(s->device);  // the kernels' attributes
    EllRun R{};
    R.g = s->ell;
    R.n = s->n;
    R.s = (int8_t*)s->state[s->cur];
    R.key = make_key(s->seed);
    R.sweep0 = (uint32_t)s->sweep;
    R.replica = s->replica;
    R.n_emcs = n_emcs;
    R.nmetro = nmetro;
    R.D = s->nbr_bound;
    R.cuts = s->d_cuts;
    R.acc = acc;
    R.status = s->d_status;
    R.wait_ns = 2000000000ull;  // 2 s
    if (s->inject_row >= 0) {   // one launch only
        R.hold = s->inject_row;
        R.wait_ns = s->inject_wait_ns;
        s->inject_row = -1;
    }
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg;
    ell_config(cfg, at, s->ell.ctas, ell_smem((size_t)s->ell.npos, s->ell.range, s->ell.rounds), s->stream);
    e = cudaLaunchKernelEx(&cfg, ell_kernel(s->ell.bonds != nullptr), R);
    s->launches++;
    s->sweep += (uint64_t)n_emcs * (uint64_t)nmetro;
    return e;
}

}  // namespace mqv
