// inplace_kernel.cuh — the in-place form of the sweep stream.
//
// The lattice stays in one buffer and a frame writes only the voxels whose
// content changes.  Each frame is three launches:
//
//   X    the voxels that lose or receive a particle along x
//   Y    ... along y
//   Z+D  ... along z, the SSA of the voxels that may react, and the decisions
//        of the next frame for every occupied voxel
//
// The decision pass (D) evaluates every occupied voxel once per frame: one
// Philox block per particle gives its x-, y- and z-words, so the move
// decisions of all three sweeps and the quiet-voxel test are made together,
// for the content the voxel has when the frame starts.  They stand for as long
// as the content does.  A sweep then has work only where a decision moves
// something: it lists the voxels that lose or receive a particle, forms their
// new contents and makes their later decisions of the frame anew.  On a lattice
// where a particle moves in 8% of its sweeps (the 256^3 multi-region cell) a
// sweep touches 8 voxels of 1024, where the record-passing forms carry all 59
// listed ones through every pass.
//
// Decisions are kept in bitmaps over the occupancy words: per axis a pair
// {moves down, moves up} (mv), and the voxels whose first reaction event may
// fall inside the frame (react).  The bit alone is the decision of a voxel of
// one particle; a voxel of more (bitmap mul) keeps its move mask (as
// decide_moves gives it) in the per-voxel array dec of the axis.
//
// Most moves are simple: a voxel's only particle goes to an empty voxel that
// receives nothing else, and nothing arrives where it came from.  The bitmaps
// of five voxels along the axis tell, so simple moves are found 32 voxels at a
// time with a few logic operations; one thread then carries out each, reading
// and writing only the species byte.  The other voxels of a sweep (shared
// targets, crowded voxels) take the general path.  In place it needs the
// contents of a voxel and of its two neighbours along the axis as the sweep
// started.  A block takes whole lines along the axis, so every voxel that a
// listed voxel exchanges particles with is listed by the same block (and none
// of them takes part in a simple move): the block first copies the listed
// voxels to the snapshot buffer, and after a barrier forms each new content
// from the snapshots and stores it.  No other block touches those voxels or
// their words.
//
// Invariants between launches: a voxel's slots are valid only where mul is set
// (a lone particle is its byte in spec, an empty voxel its clear bit in occ, and
// what the slots of either hold is left over), so whoever wants slots has them
// written first (inplace_unpack) or reads occ, mul and spec; mv of an axis is zero except
// between the pass that decides and the sweep that uses it (the sweep clears the
// words it has used); occ, mul, mv and react have no bits
// outside the lattice.  The lattice may be up to 1024 voxels long along each
// axis.
//
// What bounds it: on large lattices the instructions per bitmap word and listed
// voxel (X 53k, Y 30k, Z+D about 35k cycles per block of the 256 cubed cell: X has
// strided words); below about 100 cubed, the latency of three dependent launches,
// 25 us per frame whatever the content, where the fused stream's two win.  Blocks:
// 256 threads and up to 1024 words for X and Y (128 / 512 measured 106 us per frame
// against 98 on the 256 cubed cell, 128 against 121 on the 192 cubed one), 128 / 512
// for Z+D, whose decision pass wants its registers (7 blocks per SM).  One 16-byte
// content load per voxel of the decision pass made the 256 cubed frame 1.6 times as
// long: hence the species bytes.  us per frame in one call from frame 80 on (three
// processes within 1), fused sweep stream / this form: 256 cubed multi-region cell,
// 1 M particles 146 / 98; 192 cubed stiff network, 1 M particles 152 / 121 (194 / 137
// in its first 18 frames, while the placed particles spread); three species, K = 8, 57
// x 43 x 39 with two particles per voxel 199 / 96.  One persistent launch with grid
// barriers between the sweeps was slower throughout (1.7 and 2.7 times on the first
// two), as a barrier costs 2.7k - 4.7k cycles.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "prod_common.cuh"

namespace cellsim {

// Lines of one block.  X: the word columns a .. a + n - 1 (of the Y * Wz words of a plane) for all
// x, laid out with a pitch of 2^lw words.  Y: the words b .. b + n - 1 of every row of plane a, with
// the same pitch.  Z: the rows a .. a + n - 1 (of the X * Y rows), Wz words each.
struct LineUnit {
    uint32_t rep, a;
    uint16_t b, n, lw, pad;
};
static_assert(sizeof(LineUnit) == 16, "LineUnit is 16 bytes");

struct InplaceParams {
    ProdTables T;
    const RepDesc* reps;
    uint32_t n_rep;
    const LineUnit* units;
    uint8_t* lat;        // slots, valid for the voxels of two or more particles
    uint8_t* spec;       // [32 per word] species of the voxels of one particle
    uint8_t* snap;       // snapshots of the listed voxels of a sweep
    uint32_t* occ;       // occupancy bitmap of lat
    uint32_t* mul;       // voxels of two or more particles
    uint2* mv[3];        // per axis and word: voxels with a particle that moves down (x) / up (y)
    uint32_t* dec[3];    // per axis and voxel: the move mask of a voxel of two or more particles
    uint32_t* react;     // voxels without reservoir that may react in this frame
    const uint32_t* resv_bits;  // voxels with a reservoir species, or null
    const uint8_t* reservoir;   // per voxel, or null
    const uint8_t* region_pad;
    const uint8_t* wcode;  // per word: the region code shared by its window, or 0 (null for ensembles)
    const uint32_t* uni;   // per word: the voxels whose neighbours lie inside and share their code (null for ensembles)
    unsigned long long* counts;
    uint32_t* diag;
    // frame number f: X reads *fa = f and leaves *fb = f + 1, Y reads *fb and leaves *fa = f + 1, Z+D
    // reads *fa = f + 1 (each word is written by one launch and read by the next); explicit_frame: f
    // is `frame` and the words stay as they are
    uint32_t* fa;
    uint32_t* fb;
    uint32_t explicit_frame, frame;
    // [n_rep] the first frame of each replicate, or null: a replicate takes part in a launch of an earlier frame
    // only with the decisions of its first (replicates that stand at different frames are brought to one)
    const uint32_t* from;
    uint32_t thr_smem;     // the threshold table is staged in shared memory
    uint32_t decide_only;  // Z+D: only D, for frame f = *fa
};

constexpr int INPLACE_THREADS = 128;
constexpr int INPLACE_LINE_WORDS = 1024;  // most words of an X or Y unit (pitch included)
constexpr int INPLACE_ROW_WORDS = 512;    // ... of a Z unit
constexpr uint32_t INPLACE_MAX_EDGE = 1024;

// Launches one kernel of the form over `grid` units: axis 0, 1 the X and Y sweeps, 2 Z+D; `words` the
// most words of a unit (pitch included).
void inplace_launch(int K, int axis, uint32_t grid, uint32_t words, cudaStream_t s, const InplaceParams& P);
// Sets the kernels' shared-memory attributes for the current device.
void inplace_set_attrs();
// The region windows of a single lattice (InplaceParams::wcode, uni).
void region_windows(const uint8_t* rpad, const RepDesc& rd, uint8_t* wcode, uint32_t* uni, cudaStream_t s);
// occ, mul and spec of every replicate from its slots, and its slots from those.
void inplace_pack(int K, const InplaceParams& P, cudaStream_t s);
void inplace_unpack(int K, const InplaceParams& P, cudaStream_t s);

// View 0 (the majority species / 255) of a replicate without writing its slots.
void inplace_view(int K, const InplaceParams& P, const RepDesc& rd, uint32_t num_sms, float* out, cudaStream_t s);

}  // namespace cellsim
