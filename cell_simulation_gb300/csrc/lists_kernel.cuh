// lists_kernel.cuh — the list form of the production step.
//
// A replicate of few particles is a list of its occupied voxels, whatever the
// size of its lattice: the list form gives each replicate one block, which
// keeps that list in shared memory for every frame of a step call and never
// reads the lattice.  Between step calls the lists stay in global memory; the
// slots of the lattice are written when somebody reads them.  On the
// 512-replicate ensemble (200 A and 200 B on 32..96 cubed voxels) the other
// forms spend a frame on scanning 168 million voxels' bitmaps for 205,000
// particles.
//
// An entry is a voxel (coordinates packed in 30 bits) and its content; a hash
// table (open addressing, two slots per entry of capacity) finds the entry of a
// voxel.  A sweep is two steps between block barriers:
//
//   1. every occupied entry decides its moves along the axis; a mover finds the
//      entry of its target voxel, or makes one, and leaves its own index at the
//      target's hash slot (from below / from above)
//   2. every entry that loses or receives a particle forms its new content from
//      its own and its neighbours' contents and move masks (combine)
//
// and step 1 of the next sweep takes the new contents over.  Entries that end
// up empty stay until the list is compacted, which happens when a frame's moves
// might not fit any more.  Reactions: every occupied entry's quiet test, then an
// SSA by one warp for each voxel that may react, as in the other forms.  The
// per-voxel operations are theirs, so the lattice is the same bit for bit.
//
// A frame has room when the entries hold twice the particles (a sweep makes at most
// one entry per particle, and compaction leaves at most one per particle).  A
// replicate whose particles outgrow that stops before the frame, with its list and
// the frame's number, and tells the host; launches enqueued meanwhile leave it
// alone.  The host runs the frames it lacks over the whole GPU (device_prod.cu,
// lists_settle).
//
// What bounds it: instructions and shared-memory round trips of one block per SM;
// a frame is six dependent steps and the SSA (about 4k cycles for a sweep's first
// step, 2.5k - 3.5k for its second, 1k - 7k for the SSA on the ensemble below), and
// no DRAM traffic remains.  512 or 768 threads where an SM has one block anyway,
// else 256 so that two or three share an SM.  us per frame, fused sweep stream / lists: the
// 512 replicates above 336 / 38; 96 replicates of the stiff network with 600
// particles on 12..24 cubed voxels 43.6 / 22.7.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "prod_common.cuh"

namespace cellsim {

// ListParams::n of a replicate that has stopped: its entries and this bit, or LIST_DENSE where its state is in
// the slots (more occupied voxels than entries when the list was made).
constexpr uint32_t LIST_STOPPED = 0x80000000u;
constexpr uint32_t LIST_DENSE = 0xFFFFFFFFu;
constexpr uint32_t LIST_MAX_EDGE = 1024;
// Most frames of a launch.  The host looks between the launches of a long call whether a replicate has stopped
// (a launch's start and end take 6 us of some 10 ms).  Below 65,536, as an entry's Philox block is valid in the
// frame that its 16-bit tag names, an emptied entry keeps its tag and a launch starts every tag afresh.
constexpr uint32_t LIST_MAX_FRAMES = 1024;

struct ListParams {
    ProdTables T;
    const RepDesc* reps;
    uint8_t* lat;               // slots of the current state (read and written by pack and unpack only)
    const uint8_t* region_pad;
    uint32_t code;              // the region code of the whole lattice when it has one, else 0
    uint32_t* xyz;              // [n_rep][cap] voxels (x << 20 | y << 10 | z)
    uint8_t* cont;              // [n_rep][cap][K] contents
    uint32_t* n;                // [n_rep] entries, or LIST_STOPPED and LIST_DENSE
    uint32_t* at;               // [n_rep] the frame before which a stopped replicate stands
    uint32_t cap;               // entries per replicate, in global and in shared memory
    unsigned long long* counts;
    uint32_t* diag;
    uint32_t rep0, frame0, n_frames;  // n_frames: at most LIST_MAX_FRAMES
    uint32_t* step_out;         // the next frame's number goes here
    uint32_t* host_flag;        // host-visible word: set when a replicate has stopped
    uint32_t thr_words;         // words of the threshold table staged in shared memory (0: read from global)
};

// Shared memory of a block with `cap` entries.
size_t lists_smem(int K, uint32_t cap, uint32_t thr_words);
void lists_set_attrs(int device);
// Frames of replicates rep0 .. rep0 + grid - 1 in blocks of 256, 512 or 768 threads.
void lists_launch(int K, int threads, const ListParams& P, uint32_t grid, cudaStream_t s);
// Every replicate's list from its slots before frame P.frame0 (one with more than cap occupied voxels becomes
// LIST_DENSE), and its slots from its list; voxels_max: voxels of the largest replicate.
void lists_pack(int K, const ListParams& P, uint32_t n_rep, uint64_t voxels_max, cudaStream_t s);
void lists_unpack(int K, const ListParams& P, uint32_t n_rep, uint64_t voxels_max, cudaStream_t s);

// View 0 (the majority species / 255) of replicate 0 without writing its slots.
void lists_view(int K, const ListParams& P, const RepDesc& rd, float* out, cudaStream_t s);

}  // namespace cellsim
