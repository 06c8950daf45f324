// hpmc_kernels.h -- host-side launch interface of the sm_100a kernels.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "hpmc_device.cuh"

namespace hpmc {

// Output streams of one extraction.
struct TraverseOut {
    float4* pos;                   // x, y, z, 1 per vertex (may be null)
    float4* nrm;                   // nx, ny, nz, 0 per vertex (may be null)
    float* feedback;               // interleaved N3F_V3F, 6 floats per vertex (may be null)
    unsigned long long capacity;   // vertices the outputs can hold
    int4* dbg_cell;                // optional: x, y, z, code | k << 8 | edge << 16
    float* dbg_t;                  // optional: edge parameter t
};

// Adjoint inputs/outputs: dL/dp and dL/dn per vertex (float4, w ignored) and
// dL/df accumulated into a float lattice of the field's shape (dense, pitch
// = the field's pitches).
struct AdjointIO {
    const float4* dpos;
    const float4* dnrm;
    float* dfield;
    unsigned long long count;      // vertices to differentiate (<= vertex count)
};

// Batch-wide control block (device).
struct BatchCtrl {
    unsigned int reduce_done;     // volumes whose pyramid is complete (the last one scans)
    unsigned int work_next;       // traversal work queue: next item to hand out
    unsigned int work_done;       // traversal CTAs finished (the last one resets the queue)
    unsigned int status;          // sticky kStatus* bits of the batch
    unsigned long long total;     // vertices of all volumes
};

// Kernel view of a batch (all arrays in device memory).
struct BatchDev {
    const Volume* vols;            // per-volume descriptors (top_cached = 0)
    const CUtensorMap* tmaps;      // per-volume column tensor maps (64-byte aligned)
    const uint2* bricks;           // column bricks of the volumes with a tensor map: volume | slices << 20,
                                   // fx | fy << 9 | (first slice / column_slices) << 18
    const uint2* direct_bricks;    // of the other volumes: volume, column or block
    const uint32_t* reduce_start;  // nvol + 1: reduction chunks before volume v
    unsigned long long* vbase;     // nvol + 1: first output vertex of volume v (written by the reduction)
    uint32_t* chunk_start;         // nvol + 1: traversal work items before volume v (written by the reduction)
    BatchCtrl* ctrl;
    unsigned long long* host;      // mapped host memory (may be null): any status bit set, unused, nvol + 1 offsets
    unsigned long long capacity;   // vertices the outputs can hold
    int nvol;
    int column_slices;             // of every volume
    int stall_volume, stall_box;   // test hook (Volume::stall_box), -1: off
    int rounds;                    // traversal rounds of 32 vertices per work item
};

// Indexed-mesh extraction: scratch and outputs (device).  An "edge" below is a
// distinct edge of one group of cells of the traversal; the number of listed
// edges is Ctrl::mesh_edges.  Every edge has a vertex of its group, so a build
// of `count` vertices lists at most that many; where the device's total is
// larger (the build was replayed after its count was read), the first `count`
// vertices are welded, and the cell they end in lists at most 12 edges that
// only later vertices lie on.
constexpr uint32_t kMeshSpareEdges = 16;
struct MeshIO {
    uint32_t count;                  // soup vertices (the vertex count of the build)
    uint32_t edges;                  // entries for edges: count + kMeshSpareEdges; none is listed past them
    uint32_t* vertex;                // count: edge of each soup vertex
    uint16_t* meta;                  // count: case | vertex-in-cell << 8 (binary fields only)
    unsigned long long* keys;        // per edge: mesh_key
    uint32_t* first;                 // per edge: its smallest soup index in the group (~0: none below count)
    uint32_t* place;                 // per edge: table slot, then number of its vertex
    unsigned long long* table_keys;  // table_mask + 1 (> count, power of two)
    uint32_t* table_vals;            // right behind table_keys
    uint32_t table_mask;
    uint32_t* bits;                  // (count + 31) / 32: soup vertices that are the first on their edge
    uint32_t* scan;                  // per word of bits: set bits before it in its tile
    uint32_t* tile_sums;             // count / 65536 + 2
    unsigned int* unique;            // 1: unique vertices (mapped host or device memory)
    float4* pos;                     // unique vertices (may be null)
    float4* nrm;
    unsigned long long vcap;
    uint32_t* indices;               // one per soup vertex (may be null)
    unsigned long long icap;
};

cudaError_t launch_mesh(const Volume& V, const MeshIO& M, int normal_mode, int traverse_grid, int grid,
                        cudaStream_t st);
cudaError_t launch_classify(const Volume& V, const CUtensorMap* tmap, int max_ctas, cudaStream_t st);
cudaError_t launch_classify_batch(const BatchDev& B, int ftype, unsigned int bricks, cudaStream_t st);
cudaError_t launch_classify_batch_direct(const BatchDev& B, int ftype, unsigned int bricks, cudaStream_t st);
cudaError_t launch_reduce_batch(const BatchDev& B, unsigned int chunks, cudaStream_t st);
cudaError_t launch_traverse_batch(const BatchDev& B, const TraverseOut& O, int ftype, int normal_mode, int grid,
                                  cudaStream_t st);
int traverse_batch_blocks_per_sm();
cudaError_t launch_reduce(const Volume& V, cudaStream_t st);
cudaError_t launch_traverse(const Volume& V, const TraverseOut& O, int normal_mode, int grid,
                            cudaStream_t st);
cudaError_t launch_adjoint(const Volume& V, const AdjointIO& A, int normal_mode, int grid, cudaStream_t st);
// The TMA classifiers' dynamic shared memory on the current device: holds until
// its context is reset, so constants set it up each time they are created.
void column_smem_opt_in();
int traverse_blocks_per_sm();

}  // namespace hpmc
