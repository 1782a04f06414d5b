// Internal declarations of the batched EMCS path (batch.cu, capi.cu).
#pragma once
#include "engine.h"

namespace mqv {

// One member of a batch as the batched kernels see it.
struct BatchRep {
    ModelDev md;
    StencilDev st;              // hypercubic members
    CSRDev csr;                 // CSR members
    int lat_kind;               // MQV_LATTICE_*
    const int32_t* order;       // CSR: sites grouped by colour
    WolffDev w;                 // int8 activation rule
    Key key;
    uint32_t replica;
    uint32_t sweep0, cluster0;  // the member handle's counters when the run started
    void* s;                    // state: int8_t or float, reference site order
    uint32_t* visited;          // Wolff scratch of the member handle
    int32_t* queue;
    const unsigned long long* cuts;  // int8: the member's Metropolis cut table
    int D;                           // largest degree
    int nbr_bound;                   // int8: bound of a neighbourhood sum, the middle of the cut table
    int resident;                    // this run's EMCS are done elsewhere (batch_resident, batch_bits, ...), not in the graphs
    // labelling in bit tiles (wolff_tile.cuh): words per x-line, tiles in y and
    // z, their number (0: the lattice is labelled site by site), scratch
    int tl_nw, tl_ny, tl_nz, tl_tiles;
    int* tl_forest;             // [tiles * units * 32] global parents of local roots
    unsigned short* tl_lab;     // [tiles * units * 32] local root of every run
    // [tiles * units] candidate and x-bond words, first run of every unit
    uint32_t *tl_cand, *tl_xb, *tl_base;
};

// One cluster of a run: EMCS e_off after the device counter, cluster c of
// ncluster, and what is added to its serial (single handles).
struct ClusterStep {
    uint32_t e_off, serial_add;
    int ncluster, c;
};

// Units (32-site words of an x-line, one thread each) of a tile in y, in 3D
constexpr __host__ __device__ int tile_ty3(int units) { return units >= 256 ? 16 : 8; }

// Tiles of `units` units that cover a lattice (n = 0: not labelled in tiles:
// CSR graphs, one- and four-dimensional lattices, ids beyond 31 bits).
struct TileShape {
    int nw = 0, ny = 0, nz = 0, n = 0;
    size_t bytes(int units) const { return (size_t)n * units * (32 * 4 + 32 * 2 + 3 * 4); }
};
inline TileShape tile_shape(int lat_kind, int dim, int len, int units)
{
    TileShape t;
    if (lat_kind != MQV_LATTICE_HYPERCUBIC || dim < 2 || dim > 3) return t;
    const int ty = dim == 2 ? units : tile_ty3(units), tz = units / ty;
    t.nw = (len + 31) / 32;
    t.ny = (len + ty - 1) / ty;
    t.nz = dim == 3 ? (len + tz - 1) / tz : 1;
    const int64_t n = (int64_t)t.nw * t.ny * t.nz;
    if (n * units * 32 >= (int64_t)1 << 31) return TileShape{};
    t.n = (int)n;
    return t;
}
inline int64_t tile_lattice_units(int dim, int len)
{
    return (int64_t)((len + 31) / 32) * len * (dim == 3 ? len : 1);
}
// Units per tile and lanes per unit for so many units in all.
struct TileConfig {
    int units, lanes;
};
TileConfig tile_config(int64_t units);

// Sites of a member's lattice.
__host__ __device__ __forceinline__ int64_t rep_sites(const BatchRep& R)
{
    return R.lat_kind == MQV_LATTICE_HYPERCUBIC ? R.st.n : R.csr.n;
}

// Device counters of a run: EMCS done, first EMCS of the current chunk
// (measurement slot = e - ebase).
struct BatchCtr {
    uint32_t e;
    uint32_t ebase;
};

constexpr int kBatchMetroThreads = 256;

// Device tables and shapes the launchers need.  Colour c's work is the
// concatenation over members of their colour-c sites, each member's count
// ccount[r * ncol + c] padded to whole warp blocks of kAccSites sites:
// prefix + c * (nrep + 1) holds the padded prefix sums, block_rep +
// block_off[c] the first member of each CTA's first warp block,
// cbegin[r * ncol + c] member r's offset into its colour order.
struct BatchLaunch {
    const BatchRep* reps;
    int nrep;
    int f32;                     // float members (else int8)
    int stencil_symd;            // float: the components of every member, all on hypercubic lattices (else 0)
    int potts_octets;            // int8: every member not resident is a Potts stencil in octets
    int ncol;                    // colours of the member with the most
    const int64_t* prefix;       // [ncol][nrep + 1]
    const int32_t* block_rep;    // [sum of blocks]
    const int32_t* cbegin;       // [nrep][ncol]
    const int32_t* ccount;       // [nrep][ncol] sites of each colour
    const int* block_off;        // host: [ncol] offsets into block_rep
    const int* blocks;           // host: [ncol] blocks of each colour
    const int64_t* total;        // host: [ncol] padded work items of each colour
    // measurement: member r's sites are split over meas_prefix[r + 1] -
    // meas_prefix[r] CTAs (about 4096 sites each); meas_rep[c] is CTA c's member
    const int32_t* meas_prefix;  // [nrep + 1]
    const int32_t* meas_rep;     // [meas_blocks]
    int meas_blocks;
    // labelling in bit tiles: tiles of member r from tile_prefix[r], tile_rep[t]
    // the member of tile t
    const int32_t* tile_prefix;  // [nrep + 1]
    const int32_t* tile_rep;     // [tiles]
    int tiles;
    TileConfig tile;
    // site-level work (every site of every other member) for the labelling Wolff
    const int64_t* site_prefix;  // [nrep + 1]
    const int32_t* site_block_rep;
    int64_t total_sites;
    int site_blocks;
    void* ccl_seeds;             // [nrep] seeds of the labelling Wolff
    int wolff_ccl;               // clusters by labelling (1) or by one CTA's breadth-first growth (0)
    BatchCtr* ctr;
    long long* acc;              // slot-major accumulators (int64, or FP64 in the same words)
    int32_t* csize;              // cluster sizes: (slot * ncluster + c) * nrep + r
};

// one EMCS, e_off after the device counter; batch_launch_tick advances it
cudaError_t batch_launch_emcs(const BatchLaunch& b, cudaStream_t st, int ncluster, int nmetro, uint32_t e_off);
cudaError_t batch_launch_tick(const BatchLaunch& b, cudaStream_t st, uint32_t count);
void tile_bind(BatchRep& r, const TileShape& t, int units, void* scratch);
// the three launches of one cluster labelled in bit tiles (every tiled member)
cudaError_t launch_tile_cluster(const BatchLaunch& b, cudaStream_t st, const ClusterStep& k);
// EMCS e0 .. e0 + count - 1 of the resident members order[0 .. nres) (the
// largest with max_n sites), measurement slots from slot0 (smem_emcs.cu)
cudaError_t batch_launch_resident(const BatchLaunch& b, cudaStream_t st, const int32_t* order, int nres, size_t smem,
                                  uint32_t e0, int slot0, int count, int ncluster, int nmetro, int device);
// the same for Ising-type members held as bit planes (bits_emcs.cu)
cudaError_t batch_launch_bits(const BatchLaunch& b, cudaStream_t st, const int32_t* order, int nmem, size_t smem,
                              uint32_t e0, int slot0, int count, int ncluster, int nmetro, int device);
// the same for members held by clusters of `ctas` CTAs (cluster_emcs.cu)
cudaError_t batch_launch_cluster(const BatchLaunch& b, cudaStream_t st, const int32_t* order, int nmem, int ctas,
                                 uint32_t e0, int slot0, int count, int ncluster, int nmetro);
int cluster_ctas(int64_t n);
bool cluster_launchable(int ctas);
cudaError_t batch_launch_chunk_start(const BatchLaunch& b, cudaStream_t st, uint32_t e);
cudaError_t batch_launch_finalize(const BatchLaunch& b, cudaStream_t st, int nslots, double* out);
// raw sums of the chunk's slots -> samples[r][e0 + slot][4] (n_total EMCS per member)
cudaError_t batch_launch_samples(const BatchLaunch& b, cudaStream_t st, int nslots, int e0, int n_total,
                                 double* samples);
// replica exchange of the step's disjoint pairs ([npairs][2] member ids) from
// the energies in measurement slot `slot`; perm/flags as batch_temper describes
cudaError_t batch_launch_temper(const BatchLaunch& b, cudaStream_t st, int slot, const int32_t* pairs, int npairs, uint32_t step,
                                uint64_t seed, double en_min, double en_max, int32_t* perm, int32_t* flags);
// kernel launches of one EMCS (the counter tick of a graph apart)
inline uint64_t batch_launches_per_emcs(const BatchLaunch& b, int ncluster, int nmetro)
{
    int live = 0;
    for (int c = 0; c < b.ncol; ++c) live += b.total[c] > 0;
    // label, hook, flip of the tiled members; seed, local, hook, halve, flip of the others
    const uint64_t ccl = (b.tiles > 0 ? 3ull : 0ull) + (b.site_blocks > 0 ? 5ull : 0ull);
    return (uint64_t)ncluster * (b.wolff_ccl ? ccl : 1ull) + (uint64_t)nmetro * (uint64_t)live +
           (b.meas_blocks > 0 ? 1ull : 0ull);
}

}  // namespace mqv
