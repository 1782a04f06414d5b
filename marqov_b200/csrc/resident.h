// A chunk of EMCS of one lattice held in a CTA's shared memory
// (smem_emcs.cu, bits_emcs.cu).
#pragma once
#include "batch.h"

namespace mqv {

struct ResidentRun {
    ModelDev m;
    StencilDev st;  // the lattice in its global layout (split rows or not)
    WolffDev w;
    Key key;
    uint32_t replica, sweep0, cluster0;  // counters of the chunk's first EMCS
    int n_emcs, ncluster, nmetro, D, runs;  // D: middle of the cut table
    const unsigned long long* cuts;
    int8_t* state;      // global state, read at the start and written at the end
    long long* acc;     // measurement accumulators of the first EMCS (zeroed), or NULL
    int64_t acc_e;      // stride between EMCS (long longs)
    int32_t* csize;     // cluster size of the first cluster
    int64_t csize_e;    // stride between EMCS
    int64_t csize_c;    // stride between the clusters of one EMCS
};

#ifdef __CUDACC__
// Member r of a batch: EMCS e0 .. e0 + count - 1 of the run, measurement slots
// slot0 .. (`runs` is left to the caller).
__device__ __forceinline__ void resident_member(ResidentRun& R, const BatchRep& B, int r, int nrep, uint32_t e0,
                                                int slot0, int count, int ncluster, int nmetro, long long* acc,
                                                int32_t* csize)
{
    R.m = B.md;
    R.st = B.st;
    R.w = B.w;
    R.key = B.key;
    R.replica = B.replica;
    R.sweep0 = B.sweep0 + e0 * (uint32_t)nmetro;
    R.cluster0 = B.cluster0 + e0 * (uint32_t)ncluster;
    R.n_emcs = count;
    R.ncluster = ncluster;
    R.nmetro = nmetro;
    R.D = B.nbr_bound;
    R.cuts = B.cuts;
    R.state = (int8_t*)B.s;
    R.acc = acc + ((size_t)slot0 * nrep + r) * kAccStride;
    R.acc_e = (int64_t)nrep * kAccStride;
    R.csize = csize + (size_t)slot0 * ncluster * nrep + r;
    R.csize_e = (int64_t)ncluster * nrep;
    R.csize_c = nrep;
}
#endif

// Ising-type lattices as bit planes (bits_emcs.cu): whether the handle's
// model and lattice are of that kind and fit one CTA's shared memory (with
// room for clusters when asked).
bool bits_fits(const Sim* s, bool clusters);
size_t bits_smem(const Sim* s, bool clusters);
cudaError_t launch_bits_emcs(const ResidentRun& R, bool bonds, cudaStream_t st, int device);

}  // namespace mqv
