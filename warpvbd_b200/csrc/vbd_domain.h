// Persistent mode, fp64: the mesh divided into one domain per thread block
// (vbd_domain.cu).
#pragma once
#include <cuda_runtime.h>

#include "vbd_internal.h"
#include "vbd_persist.h"

namespace vbd {

// A domain's vertices have local ids: its own solved vertices colour by
// colour, then the halo (other domains' solved vertices that share a tet with
// an own one) colour by colour, then the unsolved vertices of its tets.
struct DomInfo {
  int env;           // its environment
  int nd, rank;      // domains of the environment, and this one's number
  int lbase;         // first entry of the domain in DomDev::local
  int nown, nloc;    // own vertices; all local vertices
  int rbase, nrec;   // its records: from DomDev::rec_id (kDomRecords) or in DomDev::rec
  int tbase, ntets;  // its tets in DomDev::tet_slot (those whose owner is its own)
  int qbase, nchunk;   // its chunks
  int cbase, ncolors;  // its colours
  int pbase;           // the environment's posts in DomDev::post: [2][nd]
  int nsave;           // kDomSave: its vertices of the first colour
  int flags;           // kDomRecords, kDomMeta, kDomSave
};

// What a block stages in shared memory beside the positions (else it reads
// global memory): the records; the chunks and DomDev::local.  kDomSave (all of an
// environment's domains or none): room for the positions of the first colour,
// which its next sweep starts on before the convergence test's answer is there.
constexpr int kDomRecords = 1, kDomMeta = 2, kDomSave = 4;

// One colour of one domain.
struct DomColor {
  int chunk_begin, chunk_end;  // the domain's chunks, counted from its first
  int halo_begin, halo_end;    // local ids of the colour's halo vertices
};

// 32 / TPV own vertices of one colour: local ids [lbegin, lend).  Lane l of its
// warp takes slots l / (32 / TPV), + TPV, ... of vertex l % (32 / TPV): the eight
// lanes that share a wavefront of 16-byte loads then visit like slots of
// neighbouring vertices.
struct DomChunk {
  int block, steps;  // SELL-32 blocks, as ChunkInfo
  int lbegin, lend;
};

struct DomDev {
  // block b runs domain first[work[b].x] + work[b].y, with `first` the array for
  // the group size work[b].z (1, or more); without work, domain b
  const int4* work;
  const int* first_single;
  const int* first_split;
  const DomInfo* dom;
  const DomColor* color;
  const DomChunk* chunk;
  const ushort4* slot;       // (n0, n1, n2, 4 x record + place), local ids
  const int2* local;         // (renumbered vertex id, or its complement when other domains
                             // read the vertex; incident tets)
  const int* rec_id;         // staged records: places in the environment's table
  const double4* rec;        // records read from global memory, three double4 each
  const int4* tet_slot;      // owner slot of every tet, local ids
  const int* tet_owner;      // its owner's local id
  ulonglong2* mail;          // [vertices][3]: (coordinate bits, tag)
  ulonglong2* post;          // (value, tag)
  unsigned* abort;           // the number of the last step in which a wait expired
  unsigned seq;              // number of this step, 1 to 2^28 - 1: tags do not repeat
  int grid_sync;             // every domain waits for every other between colours
};

constexpr int kDomMaxBlocks = 192;  // domains of an environment at most
constexpr int kDomMaxColors = 256;  // as the colouring's limit
// Threads of a block at most; one block per SM.
constexpr int kDomMaxThreads = 512;

// Dynamic shared memory of a domain's block: positions, records, chunks and
// DomDev::local entries, saved positions, each part only when its flag is set.
__host__ __device__ inline size_t dom_smem_records(int nloc) {
  return ((size_t)nloc * 24 + 15) / 16 * 16;
}
__host__ __device__ inline size_t dom_smem_meta(int nloc, int nrec, int flags) {
  return dom_smem_records(nloc) + ((flags & kDomRecords) ? (size_t)nrec * 96 : 0);
}
__host__ __device__ inline size_t dom_smem_save(int nloc, int nrec, int nchunk, int flags) {
  return dom_smem_meta(nloc, nrec, flags) +
         ((flags & kDomMeta) ? (size_t)nchunk * 16 + (size_t)nloc * 8 : 0);
}
inline size_t dom_smem(int nloc, int nrec, int nchunk, int nsave, int flags) {
  return dom_smem_save(nloc, nrec, nchunk, flags) + ((flags & kDomSave) ? (size_t)nsave * 24 : 0);
}
// Largest dynamic shared memory a domain may take: 227 KB less the kernel's
// static arrays.
constexpr size_t kDomMaxSmem = 227 * 1024 - 6400;

// Resident blocks per SM (cluster = 1) or resident clusters on the device; split:
// of a launch with environments split over several blocks.
cudaError_t dom_occupancy(int material, int tpv, int threads, size_t smem, int cluster,
                          bool split, int* out);

// One launch of a time step: n_blocks blocks, co-resident as a whole
// (cooperative) or cluster by cluster.  Writes iters, status and the state of
// the environments it runs.
cudaError_t launch_domain(int material, int tpv, int threads, const DevMesh& m,
                          const StepParams& p, const DomDev& d, const double* tol_env,
                          const PersistLimits& lim, int n_blocks, int cluster, bool cooperative,
                          size_t smem, cudaStream_t s);

}  // namespace vbd
