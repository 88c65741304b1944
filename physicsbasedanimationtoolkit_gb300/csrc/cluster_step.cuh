// A whole time step of a mesh in one thread-block cluster (no counterpart in the reference, which
// launches one kernel per colour, gpu/impl/vbd/Integrator.cu:82-103).
//
// The mesh's vertices are split into P spatially compact parts, one per block of the cluster.  A block
// keeps the current positions of its own vertices and of their neighbours in other parts (the halo) in
// shared memory for the whole step, solves its own vertices colour by colour, and stores a new position
// into the shared memory of every block that holds the vertex as halo (st.async, counted by that
// block's barrier of the colour).  A colour ends when the block's own vertices are solved and its halo
// of that colour has arrived: no launch, no trip through L2 and no cluster-wide barrier lies between
// two colours.  The solves' tables (entries, neighbours, incidences) are laid out as one contiguous
// tile per 32 vertices of a (part, colour); a producer warp streams the tiles into a ring in shared
// memory with bulk copies, ahead of the solves that read them, or once per step when they all fit.
//
// One launch carries every mesh of a batch: cluster m is mesh m (larger meshes first), and the
// hardware starts clusters as blocks become free.
//
// Why a remote store never overwrites a position that is still to be read: only neighbours read a
// vertex b, and b's next solve reads each of them.  A neighbour a in another block is read at its latest
// iterate, which its block sends after the solve in which a read b; so b's solve, and the store after
// it, follow every read of b's old position.  The same holds for the phase of a colour's barrier: bytes
// of the next iteration are sent only after the block has passed this iteration's wait.
//
// What a block reads from global memory inside a substep goes to L2 (the acquire of other blocks' positions
// empties L1), so the positions damping needs are in shared memory too: a 5,040-vertex Chebyshev step of
// 2 x 15 damped iterations took 126 us with them, 137 us without.
//
// Every wait has a time limit.  Asking for a tile as a warp costs a vote per group where tiles are streamed (4
// to 5 us of that step); with one warp waiting for the halo, and before the block's barrier, the steps take
// 124 us (that one), 58.7 (1331 vertices) and 24.0 (27 vertices) among others.
//
// What bounds it: with a few solves per part and colour, the chain of one vertex solve (about 300
// instructions of one warp, 0.8 us) times the colours; with many, shared memory (with three 16-byte reads per
// incidence: L1 at 68 % with 272 vertices per block and colour, issue at 44 %).  A first version with a
// cluster barrier per colour and tables read from global memory took 1.6 us per colour where this one
// takes 1.1: the barrier's acquire empties L1, so that every table read after it went to L2.
// 20 iterations without acceleration, colour launches -> one cluster: 27 vertices 113 -> 62 us, 1331
// vertices 285 -> 169 us, 4913 vertices 290 -> 220 us (244 with three edge vectors read per incidence
// instead of four per pair); 48 meshes of 27 to 512 vertices 795 (persistent tickets) -> 187 us.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "vbd_kernels.cuh"

namespace pbgb {

// One solved vertex of a tile.  A tile is kClusterTileVertices entries (unused ones have vertex -1),
// then, each array from a 16-byte boundary, the neighbours (slot, bit 31: lower colour; K as bits), the
// pairs of incidences (kappa, sigma of each), the pairs' slot words and the copies of the vertices'
// positions in other blocks (rank << 16 | slot there).  Offsets count from the tile's start.
struct __align__(16) ClusterEntry
{
    int32_t vertex;
    int32_t solve; // solve-list entry (the tape's order)
    uint32_t nbr;  // offset in 8-byte units | count << 16
    uint32_t pair; // offset in 16-byte units | count << 16
    uint32_t slot; // slot among the part's local vertices | copies << 16
    uint32_t words; // slot words, copies: offsets in 4-byte units, the second << 16
    float diag;     // SweepParams::diag
    int32_t pad;
};

int constexpr kClusterTileVertices = 32;

struct ClusterStepParams
{
    SweepParams sweep; // step constants
    SubstepParams sub;
    float const* __restrict__ omega;         // Chebyshev weight of each iteration
    int32_t const* __restrict__ partPtr;     // parts + 1: offsets into partVertex
    int32_t const* __restrict__ partOwned;   // own vertices of each part (they come first)
    uint32_t const* __restrict__ partVertex; // local vertices; bit 31: never solved
    int2 const* __restrict__ partColor;      // part x colour: vertices solved, halo vertices received
    int32_t const* __restrict__ partTile;    // parts + 1: tiles of each part, colours in order
    int2 const* __restrict__ tiles;          // offset in 16-byte units, bytes
    unsigned char const* __restrict__ tileData;
    int32_t nColors;
    int32_t iterations;
    int32_t substeps;
    int32_t localCapacity; // largest part's local vertices (the shared-memory layout of every block)
    int32_t ownedCapacity; // largest part's own vertices
    int32_t slabPerWarp;   // staged neighbours of the warp that stages the most
    int32_t stages;        // ring slots
    int32_t stageBytes;    // largest tile, a multiple of 128
    long long waitNs;      // time limit of one wait
    int32_t poison;        // tile of the first block (counted over the step) that never arrives (tests of the limit); -1: none
    // Recording (REC): the tape of the substep's slot, advanced by its stride per substep.
    float4* __restrict__ tapeX;   // iterates X_0 .. X_K, nV each
    float4* __restrict__ tapeRaw; // Chebyshev: raw sweep results, nV each
    float4* __restrict__ tapeH;   // inverse Newton matrices, 2 nFree per iteration
    float4* __restrict__ tapeS;   // start positions, velocities, previous velocities
    int32_t tapeIterations;       // iterations a slot holds
    int32_t nFree;
};

// A tile's size, so that its offsets fit their fields.
size_t constexpr kClusterMaxTile = 128 * 1024;
// Blocks of a cluster (a power of two up to 16), solving warps of a block and ring slots the step may
// use (one more warp streams the tiles).
int constexpr kClusterMaxBlocks = 16;
int constexpr kClusterMaxWarps  = 16;
int constexpr kClusterMaxStages = 64;
// Local vertices a part may have (slots are 15 bits in the neighbour records and 16 in the sends).
int constexpr kClusterMaxLocal = 32767;
// Dynamic shared memory of a block.
size_t constexpr kClusterMaxBytes = 226 * 1024;
// (with p.sweep.kD set)
size_t cluster_step_smem(ClusterStepParams const& p, int warps, bool chebyshev);
// Launches nMeshes clusters of `blocks` blocks.
cudaError_t launch_cluster_step(ClusterStepParams const& p, int lanes, int warps, int blocks, int nMeshes, bool chebyshev, bool record, cudaStream_t s);
// Clusters of that shape the device runs at once (0: it cannot run), with the kernel's attributes set
// on the current device.
int cluster_step_resident(int lanes, int warps, int blocks, size_t smem, bool chebyshev, bool record);

} // namespace pbgb
