// device_ref.cu — reference-RNG (bit-parity) form of the RDME timestep.
//
// Reproduces the reference shaders' arithmetic exactly (res/shader/rdme.wgsl,
// cme.wgsl, final_stage.wgsl, random.wgsl) in a canonical serial order: voxels
// in linear index order, slots in index order (the reference's own GPU order
// is nondeterministic because of its spin locks and CAS slot insertion).
//
// Directions depend only on the source lattice, so each destination voxel can
// assemble its slots on its own, in serial order: arrivals from the -x, -y, -z
// neighbours, its own departures, arrivals from the +z, +y, +x neighbours,
// each arrival into the lowest free slot.  This equals the serial order when
// no arrival can be rejected; when max(occupancy, nonzero slots) + arrivals >
// K for some voxel (`contended`), a one-thread kernel redoes the frame's
// diffusion in serial order with the capacity rule.
//
// cs_step runs the sparse form on single (in-place) state buffers.  A block
// takes a range of words of the voxel bitmaps and lists their voxels in shared
// memory, so every lane has a voxel however sparse the lattice, and no list
// passes through global memory.  Three launches per frame:
//   ref_sp_directions   over act (voxels holding a particle, a non-zero
//                       occupancy or a non-zero species count): the direction
//                       of every particle from PCG(itime + x%y + z + slot
//                       index) (rdme.wgsl:138-226); voxels with a departure
//                       store their directions and a snapshot of their slots
//                       and set their `dep` bit; every departure counts one
//                       arrival at its destination, sets both voxels' `touch`
//                       bits and raises `contended` when the destination could
//                       overflow.
//   ref_sp_move         not contended: over touch, the gather above, in place,
//                       with the species of arriving particles read from their
//                       sources' snapshots; contended: one thread of one
//                       block, the serial diffusion, in place.
//   ref_sp_cme          over act and touch: one-event reaction test, rewrite
//                       with rollback, stable compaction (final_stage.wgsl:25-33),
//                       species-count deltas reduced per block; the next
//                       frame's act words.
// Occupancy and the concentration row (68 bytes at 16 species) of nearly every
// voxel are what its slots say; such a voxel is `tidy`, and the passes neither
// read nor write the two for it: they are written when somebody reads them.
// A voxel stops being tidy when a reaction leaves a count that its slots
// cannot show (below zero, or skipped for a reservoir species).  A tidy voxel
// with one particle fires with a probability that depends on the species
// alone, tabulated by the same operations in the same order; the others sum
// only reactions whose reactants are all present (the rest add zeros).
//
// What bounds it: up to 64 cubed three launch latencies (40 cubed with 3,000
// particles 15.3 us per frame, 37.2 with six launches, two of them list
// compactions, and the rows read and written throughout); past that the
// scattered accesses per listed voxel (100 cubed with 40,000 24.2, before
// 51.9; 160 cubed with 200,000 47.1, before 84.6).  Calls of 20 frames and a
// view of 128 cubed with 22,000 particles: 989 -> 424 us; of 10 frames and a
// view of 256 cubed with 1 M: 2,856 -> 1,657 us (1,780 and 2,030 with
// the reaction networks of two other seeds).
//
// A voxel in neither act nor touch holds no particle and no species count, its slots
// are compacted and its conc[v][0] is already 1, so the reaction pass leaves
// it unchanged unless its first uniform is 0: r1 = UniformFloat(PCG(itime +
// x*y + z)) is 0 exactly when the seed is 0 (PCG and the xorshift are
// bijections that fix 0), and r1 <= 1 - exp(-0 * tau) = 0 then fires the
// selection.  Pass 1 puts those voxels (x*y + z = -itime mod 2^32) in
// touch.  The first frame after an upload, and every frame of a model
// with a reaction without reactants (non-zero propensity in every voxel), run
// the reaction pass over every voxel.
//
// The allocation-free entry point (cs_ref_frame_noalloc) runs the dense form
// of the same frame on caller-owned ping-pong buffers: five launches of one
// thread per voxel (ref_directions, ref_gather, ref_serial_copy, ref_serial,
// ref_cme), the per-voxel operations shared with the sparse form.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "cuda_check.h"
#include "devmath.cuh"
#include "views.cuh"
#include "internal.h"

namespace cellsim {

enum { DIAG_SPILL = 0, DIAG_OCC_RANGE = 1, DIAG_SLOW_STEPS = 2, DIAG_ROLLBACKS = 3, DIAG_FIRED = 4, DIAG_N = 8 };

struct RefParams {
    uint32_t X, Y, Z, K, S1, R, NR;
    uint32_t YZ;
    uint64_t V;
    float tau;
    const float* P;            // [NR][NR][S1]
    const int32_t* stoich;     // [R+1][S1]
    const uint32_t* reactants; // [R+1][3]
    const float* rates;        // [R+1]
    const uint8_t* regions;    // [V]
    const uint8_t* reservoir;  // [V]
};

// State of a reference-RNG handle: one in-place copy of the lattice (slots,
// occupancy, concentrations) and the bitmaps and scratch of the sparse form.
struct DeviceRef {
    int device = 0;
    cudaStream_t stream = nullptr;
    RefParams p{};
    DevBuf<uint8_t> slots;
    DevBuf<uint32_t> occ;
    DevBuf<int32_t> conc;
    DevBuf<uint8_t> regions, reservoir, dirs, snap;
    DevBuf<float> P, rates;
    DevBuf<int32_t> stoich, stat;
    DevBuf<uint32_t> reactants, diag, flag, itimes;
    DevBuf<uint32_t> act_bm, touch_bm, dep_bm, tidy_bm, same_bm, uses, arrivals;
    DevBuf<float> fire1;
    DevBuf<int32_t> sample_ring;
    int sms = 1, smem_optin = 0;
    bool finite = true;         // every rate is finite
    bool one_block = false;     // the frames of a call run in one block (ref_choose_form)
    bool rows_stale = false;    // frames have run since the tidy voxels' rows were written
    bool dense_next = true;   // the next reaction pass visits every voxel (first frame after an upload)
    bool dense_always = false;  // a reaction without reactants: every voxel may fire in every frame
    ~DeviceRef() {
        if (stream) cudaStreamDestroy(stream);
    }
};

// ------------------------------------------------------------------ kernels

__device__ __forceinline__ float ref_prob(const RefParams& p, uint32_t a, uint32_t b, uint32_t q) {
    return __ldg(p.P + ((size_t)a * p.NR + b) * p.S1 + q);
}

// rdme.wgsl:138-191 (probability vector), :212-226 (draw), :91-130 (edges).
__device__ int ref_decide(const RefParams& p, uint64_t v, uint32_t x, uint32_t y, uint32_t z, uint32_t q,
                          uint32_t i_part, uint32_t itime) {
    const uint8_t* reg = p.regions;
    uint32_t sr = reg[v];
    float pv[6];
    pv[0] = (x > 0u) ? ref_prob(p, sr, reg[v - p.YZ], q) : 0.0f;
    pv[1] = (x < p.X - 1u) ? __fadd_rn(pv[0], ref_prob(p, sr, reg[v + p.YZ], q)) : pv[0];
    pv[2] = (y > 0u) ? __fadd_rn(pv[1], ref_prob(p, sr, reg[v - p.Z], q)) : pv[1];
    pv[3] = (y < p.Y - 1u) ? __fadd_rn(pv[2], ref_prob(p, sr, reg[v + p.Z], q)) : pv[2];
    pv[4] = (z > 0u) ? __fadd_rn(pv[3], ref_prob(p, sr, reg[v - 1], q)) : pv[3];
    pv[5] = (z < p.Z - 1u) ? __fadd_rn(pv[4], ref_prob(p, sr, reg[v + 1], q)) : pv[4];
    uint32_t xmody = (y == 0u) ? 0u : (x % y);  // WGSL: e1 % 0 == 0
    float r = d_uniform_float(d_pcg(itime + xmody + z + i_part));
    int d = 0;
    while (d < 6 && r > pv[d]) d++;
    switch (d) {
        case 0: return (x == 0u) ? 6 : 0;
        case 1: return (x == p.X - 1u) ? 6 : 1;
        case 2: return (y == 0u) ? 6 : 2;
        case 3: return (y == p.Y - 1u) ? 6 : 3;
        case 4: return (z == 0u) ? 6 : 4;
        case 5: return (z == p.Z - 1u) ? 6 : 5;
        default: return 6;
    }
}

// ref_decide with the voxel's region codes loaded once for all its particles (rn: own, x-1, x+1,
// y-1, y+1, z-1, z+1; entries past the lattice edge are not read) and the probability table at Pt
// (shared memory when it fits): the same sums and the same draw.
__device__ __forceinline__ int ref_decide_rn(const RefParams& p, const float* Pt, const uint32_t (&rn)[7], uint32_t x,
                                             uint32_t y, uint32_t z, uint32_t q, uint32_t i_part, uint32_t itime) {
    const size_t row = (size_t)rn[0] * p.NR;
    auto prob = [&](uint32_t b) -> float { return Pt[(row + b) * p.S1 + q]; };
    float pv[6];
    pv[0] = (x > 0u) ? prob(rn[1]) : 0.0f;
    pv[1] = (x < p.X - 1u) ? __fadd_rn(pv[0], prob(rn[2])) : pv[0];
    pv[2] = (y > 0u) ? __fadd_rn(pv[1], prob(rn[3])) : pv[1];
    pv[3] = (y < p.Y - 1u) ? __fadd_rn(pv[2], prob(rn[4])) : pv[2];
    pv[4] = (z > 0u) ? __fadd_rn(pv[3], prob(rn[5])) : pv[3];
    pv[5] = (z < p.Z - 1u) ? __fadd_rn(pv[4], prob(rn[6])) : pv[4];
    uint32_t xmody = (y == 0u) ? 0u : (x % y);  // WGSL: e1 % 0 == 0
    float r = d_uniform_float(d_pcg(itime + xmody + z + i_part));
    int d = 0;
    while (d < 6 && r > pv[d]) d++;
    switch (d) {
        case 0: return (x == 0u) ? 6 : 0;
        case 1: return (x == p.X - 1u) ? 6 : 1;
        case 2: return (y == 0u) ? 6 : 2;
        case 3: return (y == p.Y - 1u) ? 6 : 3;
        case 4: return (z == 0u) ? 6 : 4;
        case 5: return (z == p.Z - 1u) ? 6 : 5;
        default: return 6;
    }
}

__global__ void ref_directions(RefParams p, const uint8_t* __restrict__ src, const uint32_t* __restrict__ occS,
                               const uint32_t* __restrict__ itimes, uint32_t step, uint8_t* __restrict__ dirs,
                               uint32_t* diag, uint32_t* contended) {
    uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v == 0) *contended = 0u;
    if (v >= p.V) return;
    uint32_t z = (uint32_t)(v % p.Z);
    uint32_t y = (uint32_t)((v / p.Z) % p.Y);
    uint32_t x = (uint32_t)(v / p.YZ);
    uint32_t o = occS[v];
    if (o > p.K) { atomicAdd(diag + DIAG_OCC_RANGE, 1u); o = p.K; }
    uint32_t itime = itimes[step];
    for (uint32_t s = 0; s < p.K; s++) {
        uint32_t i_part = (uint32_t)(v * p.K + s);
        uint32_t q = src[i_part];
        uint8_t d = 7;
        if (s < o && q != 0u) d = (uint8_t)ref_decide(p, v, x, y, z, q, i_part, itime);
        dirs[i_part] = d;
    }
}

__device__ __forceinline__ int64_t ref_nb_offset(const RefParams& p, int d) {
    switch (d) {
        case 0: return -(int64_t)p.YZ;
        case 1: return (int64_t)p.YZ;
        case 2: return -(int64_t)p.Z;
        case 3: return (int64_t)p.Z;
        case 4: return -1;
        default: return 1;
    }
}

__global__ void ref_gather(RefParams p, const uint8_t* __restrict__ src, const uint32_t* __restrict__ occS,
                           const int32_t* __restrict__ concS, const uint8_t* __restrict__ dirs,
                           uint8_t* __restrict__ dst, uint32_t* __restrict__ occD, int32_t* __restrict__ concD,
                           uint32_t* contended) {
    uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= p.V) return;
    const uint32_t K = p.K, S1 = p.S1;
    uint32_t z = (uint32_t)(w % p.Z);
    uint32_t y = (uint32_t)((w / p.Z) % p.Y);
    uint32_t x = (uint32_t)(w / p.YZ);
    bool has_nb[6] = {x > 0u, x < p.X - 1u, y > 0u, y < p.Y - 1u, z > 0u, z < p.Z - 1u};
    uint8_t sl[16];
    uint32_t nnz = 0, in = 0;
    for (uint32_t s = 0; s < K; s++) { sl[s] = src[w * K + s]; nnz += sl[s] != 0; }
    for (int side = 0; side < 6; side++) {
        if (!has_nb[side]) continue;
        uint64_t u = (uint64_t)((int64_t)w + ref_nb_offset(p, side));
        uint8_t want = (uint8_t)(side ^ 1);
        for (uint32_t s = 0; s < K; s++) in += dirs[u * K + s] == want;
    }
    uint32_t o = occS[w];
    uint32_t base = o > nnz ? o : nnz;
    if (base + in > K) {
        atomicOr(contended, 1u);
        return;
    }
    int32_t* cw = concD + w * S1;
    const int32_t* cs = concS + w * S1;
    for (uint32_t s = 0; s < S1; s++) cw[s] = cs[s];
    const int lower[3] = {1, 3, 5}, upper[3] = {4, 2, 0};
    for (int k = 0; k < 3; k++) {
        int want = lower[k], side = want ^ 1;
        if (!has_nb[side]) continue;
        uint64_t u = (uint64_t)((int64_t)w + ref_nb_offset(p, side));
        for (uint32_t s = 0; s < K; s++) {
            if (dirs[u * K + s] != want) continue;
            uint8_t q = src[u * K + s];
            uint32_t j = 0;
            while (sl[j] != 0) j++;
            sl[j] = q; o++; cw[q] += 1;
        }
    }
    for (uint32_t s = 0; s < K; s++) {
        if (dirs[w * K + s] < 6) {
            uint8_t q = sl[s];
            sl[s] = 0; o--; cw[q] -= 1;
        }
    }
    for (int k = 0; k < 3; k++) {
        int want = upper[k], side = want ^ 1;
        if (!has_nb[side]) continue;
        uint64_t u = (uint64_t)((int64_t)w + ref_nb_offset(p, side));
        for (uint32_t s = 0; s < K; s++) {
            if (dirs[u * K + s] != want) continue;
            uint8_t q = src[u * K + s];
            uint32_t j = 0;
            while (sl[j] != 0) j++;
            sl[j] = q; o++; cw[q] += 1;
        }
    }
    for (uint32_t s = 0; s < K; s++) dst[w * K + s] = sl[s];
    occD[w] = o;
}

__global__ void ref_serial_copy(RefParams p, const uint32_t* contended, const uint8_t* __restrict__ src,
                                const uint32_t* __restrict__ occS, const int32_t* __restrict__ concS,
                                uint8_t* __restrict__ dst, uint32_t* __restrict__ occD, int32_t* __restrict__ concD) {
    if (*contended == 0u) return;
    uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t i = t; i < p.V * p.K; i += stride) dst[i] = src[i];
    for (uint64_t i = t; i < p.V; i += stride) occD[i] = occS[i];
    for (uint64_t i = t; i < p.V * p.S1; i += stride) concD[i] = concS[i];
}

// Serial diffusion with the capacity rule (rdme.wgsl:45-88): a move into a
// voxel whose occupancy is >= K, or that has no zero slot, is rejected.
__global__ void ref_serial(RefParams p, const uint32_t* contended, const uint8_t* __restrict__ src,
                           const uint32_t* __restrict__ occS, const uint8_t* __restrict__ dirs,
                           uint8_t* __restrict__ dst, uint32_t* __restrict__ occD, int32_t* __restrict__ concD,
                           uint32_t* diag) {
    if (*contended == 0u || threadIdx.x != 0 || blockIdx.x != 0) return;
    const uint32_t K = p.K, S1 = p.S1;
    uint32_t spills = 0;
    for (uint64_t v = 0; v < p.V; v++) {
        uint32_t o = occS[v];
        if (o > K) o = K;
        for (uint32_t s = 0; s < o; s++) {
            uint64_t i = v * K + s;
            int d = dirs[i];
            if (d >= 6) continue;
            uint64_t w = (uint64_t)((int64_t)v + ref_nb_offset(p, d));
            if (occD[w] >= K) { spills++; continue; }
            uint32_t j = 0;
            while (j < K && dst[w * K + j] != 0) j++;
            if (j == K) { spills++; continue; }
            uint8_t q = src[i];
            dst[w * K + j] = q;
            occD[w] += 1u;
            concD[w * S1 + q] += 1;
            occD[v] -= 1u;
            dst[i] = 0;
            concD[v * S1 + q] -= 1;
        }
    }
    diag[DIAG_SPILL] += spills;
    diag[DIAG_SLOW_STEPS] += 1u;
}

// Coordinates of voxel v (V * K < 2^32 on this path: the reference indexes
// slots with u32, functions.wgsl:42-51).
__device__ __forceinline__ void ref_coords(const RefParams& p, uint32_t v, uint32_t& x, uint32_t& y, uint32_t& z) {
    const uint32_t t = v / p.Z;
    z = v - t * p.Z;
    x = t / p.Y;
    y = t - x * p.Y;
}

// The K (<= 16) slot bytes of one voxel held in two 64-bit registers, byte i =
// slot i, so that the reaction pass touches the slot array with one load and
// at most one store per voxel.
struct RefSlots {
    uint64_t lo, hi;
};

__device__ __forceinline__ uint32_t rs_get(const RefSlots& a, uint32_t i) {
    return (uint32_t)((i < 8u ? a.lo >> (8u * i) : a.hi >> (8u * (i - 8u))) & 0xFFull);
}

__device__ __forceinline__ void rs_set(RefSlots& a, uint32_t i, uint32_t q) {
    if (i < 8u) a.lo = (a.lo & ~(0xFFull << (8u * i))) | ((uint64_t)q << (8u * i));
    else a.hi = (a.hi & ~(0xFFull << (8u * (i - 8u)))) | ((uint64_t)q << (8u * (i - 8u)));
}

// Vector access when K is 8 or 16 and the voxel's slots are aligned to it (the library's own
// buffers always are; a caller's buffer of the allocation-free entry point may not be).
__device__ __forceinline__ RefSlots rs_load(const uint8_t* sl, uint32_t K) {
    RefSlots a{0ull, 0ull};
    const uintptr_t al = (uintptr_t)sl;
    if (K == 16u && (al & 15u) == 0u) {
        const uint4 t = *reinterpret_cast<const uint4*>(sl);
        a.lo = (uint64_t)t.x | ((uint64_t)t.y << 32);
        a.hi = (uint64_t)t.z | ((uint64_t)t.w << 32);
    } else if (K == 8u && (al & 7u) == 0u) {
        const uint2 t = *reinterpret_cast<const uint2*>(sl);
        a.lo = (uint64_t)t.x | ((uint64_t)t.y << 32);
    } else {
        for (uint32_t i = 0; i < K; i++) rs_set(a, i, sl[i]);
    }
    return a;
}

__device__ __forceinline__ void rs_store(uint8_t* sl, uint32_t K, const RefSlots& a) {
    const uintptr_t al = (uintptr_t)sl;
    if (K == 16u && (al & 15u) == 0u) {
        *reinterpret_cast<uint4*>(sl) = make_uint4((uint32_t)a.lo, (uint32_t)(a.lo >> 32), (uint32_t)a.hi,
                                                   (uint32_t)(a.hi >> 32));
    } else if (K == 8u && (al & 7u) == 0u) {
        *reinterpret_cast<uint2*>(sl) = make_uint2((uint32_t)a.lo, (uint32_t)(a.lo >> 32));
    } else {
        for (uint32_t i = 0; i < K; i++) sl[i] = (uint8_t)rs_get(a, i);
    }
}

// cme.wgsl:26-120 and final_stage.wgsl:25-33 for voxel v, in place:
// conc[v][0] = 1, the one-event test, the species-major rewrite with rollback
// and the stable compaction.  s_delta[0..S1) collects species deltas,
// s_delta[S1] fired voxels and s_delta[S1 + 1] rollbacks (block-shared).
__device__ void ref_cme_voxel(const RefParams& p, uint64_t v, uint8_t* __restrict__ slots, uint32_t* __restrict__ occ,
                              int32_t* __restrict__ conc, uint32_t itime, int32_t* s_delta) {
    const uint32_t K = p.K, S1 = p.S1, R = p.R;
    const uint32_t S = S1 - 1;
    uint32_t x, y, z;
    ref_coords(p, (uint32_t)v, x, y, z);
    int32_t* c = conc + v * S1;
    uint8_t* slp = slots + v * K;
    if (c[0] != 1) c[0] = 1;  // stored only when it changes: an unchanged row is not written back
    float total = 0.0f;
    for (uint32_t r = 1; r <= R; r++) {
        uint32_t prod = (uint32_t)c[p.reactants[r * 3]] * (uint32_t)c[p.reactants[r * 3 + 1]] *
                        (uint32_t)c[p.reactants[r * 3 + 2]];
        total = __fadd_rn(total, __fmul_rn(p.rates[r], __int2float_rn((int32_t)prod)));
    }
    const RefSlots snap = rs_load(slp, K);
    RefSlots sl = snap;
    uint32_t state = d_pcg(itime + x * y + z);
    float r1 = d_uniform_float(state);
    float fire_p = __fsub_rn(1.0f, d_expf(__fmul_rn(-total, p.tau)));
    if (r1 <= fire_p) {
        atomicAdd(&s_delta[S1], 1);
        float r2 = d_uniform_float(state + 1u);
        // selection over cum[i] = cum[i-1] + a_i, normalised for i < R (cme.wgsl:50-52,70-73)
        uint32_t i = 0;
        float run = 0.0f;
        while (i < R) {
            if (!(r2 > __fdiv_rn(run, total))) break;
            i++;
            uint32_t prod = (uint32_t)c[p.reactants[i * 3]] * (uint32_t)c[p.reactants[i * 3 + 1]] *
                            (uint32_t)c[p.reactants[i * 3 + 2]];
            run = __fadd_rn(run, __fmul_rn(p.rates[i], __int2float_rn((int32_t)prod)));
        }
        const int32_t* st = p.stoich + (size_t)i * S1;
        uint32_t j = 0;
        int32_t new_occ = (int32_t)occ[v];
        uint64_t ri = v * K;  // reservoirs[idx_lattice], cme.wgsl:80
        uint32_t resv = (ri < p.V) ? p.reservoir[ri] : 0u;
        bool rolled = false;
        for (uint32_t s = 1; s <= S && !rolled; s++) {
            if (resv == s) continue;
            int32_t d = st[s];
            c[s] = (int32_t)((uint32_t)c[s] + (uint32_t)d);
            new_occ = (int32_t)((uint32_t)new_occ + (uint32_t)d);
            if (d) atomicAdd(&s_delta[s], d);
            int32_t cc = c[s];
            while (cc > 0) {
                rs_set(sl, j, s);
                cc--;
                j++;
                if (j >= K) {
                    sl = snap;
                    for (uint32_t s2 = 1; s2 <= s; s2++) {
                        int32_t d2 = st[s2];
                        c[s2] = (int32_t)((uint32_t)c[s2] - (uint32_t)d2);
                        if (d2) atomicAdd(&s_delta[s2], -d2);
                    }
                    atomicAdd(&s_delta[S1 + 1], 1);
                    rolled = true;
                    break;
                }
            }
        }
        if (!rolled) {
            occ[v] = (uint32_t)new_occ;
            while (j < K) rs_set(sl, j++, 0u);
        }
    }
    // stable move of the non-zero slots to the front
    RefSlots out{0ull, 0ull};
    uint32_t jj = 0;
    for (uint32_t s = 0; s < K; s++) {
        const uint32_t q = rs_get(sl, s);
        if (q != 0u) rs_set(out, jj++, q);
    }
    if (out.lo != snap.lo || out.hi != snap.hi) rs_store(slp, K, out);
}

// Adds a block's species deltas, fired voxels and rollbacks to the totals.
__device__ __forceinline__ void ref_flush_block(const RefParams& p, const int32_t* s_delta, int32_t* stat, uint32_t* diag) {
    for (uint32_t s = threadIdx.x; s < p.S1; s += blockDim.x)
        if (s_delta[s]) atomicAdd(stat + s, s_delta[s]);
    if (threadIdx.x == 0) {
        if (s_delta[p.S1]) atomicAdd(diag + DIAG_FIRED, (uint32_t)s_delta[p.S1]);
        if (s_delta[p.S1 + 1]) atomicAdd(diag + DIAG_ROLLBACKS, (uint32_t)s_delta[p.S1 + 1]);
    }
}

// Dense reaction pass: one thread per voxel.
__global__ void ref_cme(RefParams p, uint8_t* __restrict__ dst, uint32_t* __restrict__ occD, int32_t* __restrict__ concD,
                        const uint32_t* __restrict__ itimes, uint32_t step, int32_t* stat, uint32_t* diag) {
    extern __shared__ int32_t s_delta[];  // [S1] + 2 counters
    for (uint32_t s = threadIdx.x; s < p.S1 + 2; s += blockDim.x) s_delta[s] = 0;
    __syncthreads();
    uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < p.V) ref_cme_voxel(p, v, dst, occD, concD, itimes[step], s_delta);
    __syncthreads();
    ref_flush_block(p, s_delta, stat, diag);
}

// ------------------------------------------------------------------ sparse form

// Bitmaps over the linear voxel index (word i holds voxels 32i .. 32i+31):
//   act    voxels that hold a particle, a non-zero occupancy or a non-zero
//          species count (s >= 1)
//   touch  voxels that gain or lose particles this frame, or whose reaction
//          seed is 0
//   dep    voxels with a departure this frame
//   tidy   voxels whose occupancy and species counts are those of their slots:
//          no pass reads or writes the two arrays for them (ref_write_rows
//          does when somebody asks for them)
//   same   voxels whose six neighbours lie in the lattice and share their region
// A block owns ranges of cw consecutive words and lists their voxels in shared
// memory; no launch keeps a list in global memory.
struct RefSparse {
    uint32_t* act;
    uint32_t* touch;
    uint32_t* dep;
    uint32_t* tidy;
    const uint32_t* same;
    uint32_t* arrivals;    // [V] particles moving into the voxel this frame (zero between frames)
    uint8_t* dirs;         // [V*K] direction codes of a voxel with a departure (7 = stays)
    uint8_t* snap;         // [V*K] slots of a voxel with a departure, as the frame started
    const uint32_t* uses;  // [S1][UW] reactions (bit r) that need species s
    const float* fire1;    // [S1] firing probability of an empty voxel (0) or of a sole particle of species q
    uint32_t W;            // bitmap words
    uint32_t cw;           // words of a range
    uint32_t UW;           // words of a reaction mask
    uint32_t finite;       // every rate is finite: a reaction that lacks a reactant adds 0
};

// A word that other blocks or threads write (global memory, or shared memory in the one-block form).
__device__ __forceinline__ uint32_t ref_word(const uint32_t* p) { return *reinterpret_cast<const volatile uint32_t*>(p); }
__device__ __forceinline__ bool bit_of(const uint32_t* bm, uint32_t v) { return (ref_word(bm + (v >> 5)) >> (v & 31u)) & 1u; }
__device__ __forceinline__ void set_bit(uint32_t* bm, uint32_t v) { atomicOr(bm + (v >> 5), 1u << (v & 31u)); }

// Byte tests on slot registers: bit 7 of byte i of the result is the answer for slot i.
__device__ __forceinline__ uint64_t bytes_nonzero(uint64_t x) {
    return (((x & 0x7F7F7F7F7F7F7F7Full) + 0x7F7F7F7F7F7F7F7Full) | x) & 0x8080808080808080ull;
}
struct RefMask {
    uint64_t lo, hi;
};
__device__ __forceinline__ RefMask rs_valid(uint32_t K) {  // the K slots
    const uint64_t b = 0x8080808080808080ull;
    return RefMask{K >= 8u ? b : b & ((1ull << (8u * K)) - 1ull), K >= 16u ? b : K > 8u ? b & ((1ull << (8u * (K - 8u))) - 1ull) : 0ull};
}
__device__ __forceinline__ uint32_t rm_count(const RefMask& m) { return (uint32_t)(__popcll(m.lo) + __popcll(m.hi)); }
__device__ __forceinline__ bool rm_any(const RefMask& m) { return (m.lo | m.hi) != 0ull; }
// the lowest marked slot (one must be)
__device__ __forceinline__ uint32_t rm_first(const RefMask& m) {
    return m.lo ? (uint32_t)(__ffsll((long long)m.lo) - 1) >> 3 : 8u + ((uint32_t)(__ffsll((long long)m.hi) - 1) >> 3);
}
__device__ __forceinline__ void rm_drop(RefMask& m) {
    if (m.lo) m.lo &= m.lo - 1ull;
    else m.hi &= m.hi - 1ull;
}
__device__ __forceinline__ RefMask rs_full(const RefSlots& a) { return RefMask{bytes_nonzero(a.lo), bytes_nonzero(a.hi)}; }
__device__ __forceinline__ uint32_t rs_count(const RefSlots& a) { return rm_count(rs_full(a)); }

// The library's own buffers: K = KT (16 or 8), vector access; KT = 0: any K.
template <int KT>
__device__ __forceinline__ RefSlots rk_load(const uint8_t* base, uint32_t v, uint32_t K) {
    if constexpr (KT == 16) {
        const uint4 t = *reinterpret_cast<const uint4*>(base + (size_t)v * 16u);
        return RefSlots{(uint64_t)t.x | ((uint64_t)t.y << 32), (uint64_t)t.z | ((uint64_t)t.w << 32)};
    } else if constexpr (KT == 8) {
        const uint2 t = *reinterpret_cast<const uint2*>(base + (size_t)v * 8u);
        return RefSlots{(uint64_t)t.x | ((uint64_t)t.y << 32), 0ull};
    } else {
        return rs_load(base + (size_t)v * K, K);
    }
}
template <int KT>
__device__ __forceinline__ void rk_store(uint8_t* base, uint32_t v, uint32_t K, const RefSlots& a) {
    rs_store(base + (size_t)v * K, KT ? (uint32_t)KT : K, a);
}

// Programmatic dependent launch between the passes of a frame: a pass lets the next one launch at
// once, stages the tables that no launch writes, and waits for the previous pass to complete (and
// its memory to be visible) before it touches anything else; without a programmatic dependency the
// wait returns at once.
__device__ __forceinline__ void ref_allow_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void ref_wait_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Each pass is a device body, run by its own launch or, on small lattices, by the one-block form
// ref_sp_frames_block.  Shared memory of a body: the range's word areas and list, then its tables.
enum : int { RW_A, RW_B, RW_C, REF_AREAS };
struct RefRange {
    uint32_t* area[REF_AREAS];  // [cw] each
    uint16_t* list;             // [32 * cw] (word << 5) | bit
    uint32_t* tmp;              // [32]
};
__host__ __device__ constexpr size_t ref_range_words(uint32_t cw) { return REF_AREAS * (size_t)cw + 16 * (size_t)cw + 32; }
__device__ __forceinline__ RefRange ref_range(uint32_t* sm, uint32_t cw) {
    RefRange r;
    for (int a = 0; a < REF_AREAS; a++) r.area[a] = sm + a * cw;
    r.list = reinterpret_cast<uint16_t*>(sm + REF_AREAS * cw);
    r.tmp = sm + (REF_AREAS + 16) * cw;
    return r;
}

// Lists the voxels of the range's words (thread t's word m is word t of the range, 0 past the
// range), in word order; every thread of the block calls it.  Returns how many there are.  The
// caller's barrier comes before the next call.
template <int NT>
__device__ __forceinline__ uint32_t ref_list(uint32_t m, const RefRange& R) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, n = (uint32_t)__popc(m);
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += u;
    }
    if (lane == 31u) R.tmp[w] = incl;
    __syncthreads();
    uint32_t at = incl - n, total = 0;
#pragma unroll
    for (int i = 0; i < NT / 32; i++) {
        const uint32_t t = R.tmp[i];
        if (i < (int)w) at += t;
        total += t;
    }
    for (; m; m &= m - 1u) R.list[at++] = (uint16_t)((threadIdx.x << 5) | (uint32_t)(__ffs((int)m) - 1));
    __syncthreads();
    return total;
}

__device__ __forceinline__ void ref_stage_P(const RefParams& p, float* s_P, uint32_t stage_P) {
    if (stage_P)
        for (uint32_t i = threadIdx.x; i < p.NR * p.NR * p.S1; i += blockDim.x) s_P[i] = p.P[i];
}

// Pass 1: directions of every particle; departures, arrival counts, touched voxels and the
// contention test.  Also marks the voxels whose reaction seed itime + x*y + z is 0 this frame.
template <int KT, int NT>
__device__ __forceinline__ void ref_sp_directions_body(const RefParams& p, const RefSparse& sp, const uint8_t* slots,
                                                       const uint32_t* occ, uint32_t itime, uint32_t* diag,
                                                       uint32_t* contended, const RefRange& R, const float* Pt) {
    const uint32_t K = KT ? (uint32_t)KT : p.K;
    const uint32_t XY = p.X * p.Y, step = gridDim.x * NT, dx = step / p.Y, dy = step - dx * p.Y;
    {
        uint32_t g = blockIdx.x * NT + threadIdx.x, x = g / p.Y, y = g - x * p.Y;
        for (; g < XY; g += step) {
            const uint32_t z = 0u - itime - x * y;  // u32 wrap, as the shader's seed arithmetic
            if (z < p.Z) set_bit(sp.touch, g * p.Z + z);
            x += dx;
            y += dy;
            if (y >= p.Y) {
                y -= p.Y;
                x++;
            }
        }
    }
    for (uint32_t w0 = blockIdx.x * sp.cw; w0 < sp.W; w0 += gridDim.x * sp.cw) {
        const uint32_t i = w0 + threadIdx.x;
        const bool own = threadIdx.x < sp.cw && i < sp.W;
        const uint32_t m = own ? sp.act[i] : 0u;
        if (own) {
            R.area[RW_A][threadIdx.x] = m ? sp.tidy[i] : 0u;
            R.area[RW_B][threadIdx.x] = m ? __ldg(sp.same + i) : 0u;
            R.area[RW_C][threadIdx.x] = 0u;  // departures
        }
        const uint32_t n = ref_list<NT>(m, R);
        for (uint32_t e = threadIdx.x; e < n; e += NT) {
            const uint32_t idx = R.list[e] >> 5, b = R.list[e] & 31u, bit = 1u << b;
            const uint32_t v = (w0 + idx) * 32u + b;
            const RefSlots sl = rk_load<KT>(slots, v, K);
            RefMask full = rs_full(sl);
            if (!(R.area[RW_A][idx] & bit)) {
                uint32_t o = occ[v];
                if (o > K) {
                    // the gather's contention test fails for this voxel whatever arrives
                    atomicAdd(diag + DIAG_OCC_RANGE, 1u);
                    atomicOr(contended, 1u);
                    o = K;
                }
                const RefMask below = rs_valid(o);  // slots past the occupancy don't move
                full.lo &= below.lo;
                full.hi &= below.hi;
            } else if (rm_any(full)) {
                // a tidy voxel's occupancy is the number of its particles, wherever they lie
                const RefMask below = rs_valid(rm_count(full));
                full.lo &= below.lo;
                full.hi &= below.hi;
            }
            if (!rm_any(full)) continue;
            uint32_t x, y, z;
            ref_coords(p, v, x, y, z);
            const uint8_t* reg = p.regions;
            uint32_t rn[7];
            rn[0] = reg[v];
            if (R.area[RW_B][idx] & bit) {
#pragma unroll
                for (int k = 1; k < 7; k++) rn[k] = rn[0];
            } else {
#pragma unroll
                for (int k = 1; k < 7; k++) rn[k] = 0u;
                if (x > 0u) rn[1] = reg[v - p.YZ];
                if (x < p.X - 1u) rn[2] = reg[v + p.YZ];
                if (y > 0u) rn[3] = reg[v - p.Z];
                if (y < p.Y - 1u) rn[4] = reg[v + p.Z];
                if (z > 0u) rn[5] = reg[v - 1];
                if (z < p.Z - 1u) rn[6] = reg[v + 1];
            }
            RefSlots dr{0x0707070707070707ull, 0x0707070707070707ull};  // 7: stays
            RefMask leave{0ull, 0ull};
            for (; rm_any(full); rm_drop(full)) {
                const uint32_t s = rm_first(full);
                const int d = ref_decide_rn(p, Pt, rn, x, y, z, rs_get(sl, s), v * K + s, itime);
                if (d >= 6) continue;
                rs_set(dr, s, (uint32_t)d);
                if (s < 8u) leave.lo |= 0x80ull << (8u * s);
                else leave.hi |= 0x80ull << (8u * (s - 8u));
            }
            if (!rm_any(leave)) continue;
            rk_store<KT>(sp.dirs, v, K, dr);
            rk_store<KT>(sp.snap, v, K, sl);
            atomicOr(&R.area[RW_C][idx], bit);
            for (; rm_any(leave); rm_drop(leave)) {
                const uint32_t w = (uint32_t)((int64_t)v + ref_nb_offset(p, (int)rs_get(dr, rm_first(leave))));
                const uint32_t before = atomicAdd(sp.arrivals + w, 1u);
                set_bit(sp.touch, w);
                const uint32_t nnz = rs_count(rk_load<KT>(slots, w, K));
                uint32_t base = nnz;
                if (!bit_of(sp.tidy, w)) {
                    const uint32_t ow = occ[w];
                    base = ow > nnz ? ow : nnz;
                }
                if ((uint64_t)base + before + 1u > K) atomicOr(contended, 1u);
            }
        }
        __syncthreads();
        if (own) {
            const uint32_t d = R.area[RW_C][threadIdx.x];
            if (d) {
                sp.dep[i] = d;
                atomicOr(sp.touch + i, d);
            }
        }
        __syncthreads();
    }
}

// Pass 2 (frames without contention): the gather of every touched voxel, in place.
template <int KT, int NT>
__device__ __forceinline__ void ref_sp_gather_body(const RefParams& p, const RefSparse& sp, uint8_t* slots, uint32_t* occ,
                                                   int32_t* conc, const RefRange& R) {
    const uint32_t K = KT ? (uint32_t)KT : p.K, S1 = p.S1;
    const RefMask valid = rs_valid(K);
    for (uint32_t w0 = blockIdx.x * sp.cw; w0 < sp.W; w0 += gridDim.x * sp.cw) {
        const uint32_t i = w0 + threadIdx.x;
        const bool own = threadIdx.x < sp.cw && i < sp.W;
        const uint32_t m = own ? ref_word(sp.touch + i) : 0u;
        if (own) {
            R.area[RW_A][threadIdx.x] = m ? sp.tidy[i] : 0u;
            R.area[RW_B][threadIdx.x] = m ? ref_word(sp.dep + i) : 0u;
        }
        const uint32_t n = ref_list<NT>(m, R);
        for (uint32_t e = threadIdx.x; e < n; e += NT) {
            const uint32_t idx = R.list[e] >> 5, b = R.list[e] & 31u, bit = 1u << b;
            const uint32_t w = (w0 + idx) * 32u + b;
            uint32_t x, y, z;
            ref_coords(p, w, x, y, z);
            const bool has_nb[6] = {x > 0u, x < p.X - 1u, y > 0u, y < p.Y - 1u, z > 0u, z < p.Z - 1u};
            // the departure words of all six sides, then the snapshots of those that left, each in flight together
            bool from[6];
#pragma unroll
            for (int s = 0; s < 6; s++) {
                const uint32_t u = has_nb[s] ? (uint32_t)((int64_t)w + ref_nb_offset(p, s)) : w;
                from[s] = has_nb[s] && bit_of(sp.dep, u);
            }
            RefSlots sl = rk_load<KT>(slots, w, K);
            RefSlots nd[6], ns[6];
            const bool leaves = R.area[RW_B][idx] & bit;
            RefSlots own_d{0x0707070707070707ull, 0x0707070707070707ull};
            if (leaves) own_d = rk_load<KT>(sp.dirs, w, K);
#pragma unroll
            for (int s = 0; s < 6; s++) {
                nd[s] = ns[s] = RefSlots{0ull, 0ull};
                if (!from[s]) continue;
                const uint32_t u = (uint32_t)((int64_t)w + ref_nb_offset(p, s));
                nd[s] = rk_load<KT>(sp.dirs, u, K);
                ns[s] = rk_load<KT>(sp.snap, u, K);
            }
            sp.arrivals[w] = 0u;
            const bool tidy = R.area[RW_A][idx] & bit;
            int32_t* const cw = conc + (size_t)w * S1;
            uint32_t o = tidy ? 0u : occ[w];
            // arrivals from the neighbour on side `s`: the particles it moves in direction s ^ 1
            auto arrive = [&](int s) {
                if (!from[s]) return;
                const uint64_t want = (uint64_t)(uint32_t)(s ^ 1) * 0x0101010101010101ull;
                RefMask mv{~bytes_nonzero(nd[s].lo ^ want) & valid.lo, ~bytes_nonzero(nd[s].hi ^ want) & valid.hi};
                for (; rm_any(mv); rm_drop(mv)) {
                    const uint32_t q = rs_get(ns[s], rm_first(mv));
                    const RefMask full = rs_full(sl);
                    const RefMask room{~full.lo & valid.lo, ~full.hi & valid.hi};
                    if (!rm_any(room)) continue;  // unreachable without contention
                    rs_set(sl, rm_first(room), q);
                    if (!tidy) {
                        o++;
                        cw[q] = (int32_t)((uint32_t)cw[q] + 1u);
                    }
                }
            };
            arrive(0);  // from -x
            arrive(2);  // from -y
            arrive(4);  // from -z
            if (leaves) {
                // direction bytes below 6 (they are at most 7)
                RefMask mv{~(own_d.lo + 0x7A7A7A7A7A7A7A7Aull) & valid.lo, ~(own_d.hi + 0x7A7A7A7A7A7A7A7Aull) & valid.hi};
                for (; rm_any(mv); rm_drop(mv)) {
                    const uint32_t s = rm_first(mv), q = rs_get(sl, s);
                    rs_set(sl, s, 0u);
                    if (!tidy) {
                        o--;
                        cw[q] = (int32_t)((uint32_t)cw[q] - 1u);
                    }
                }
            }
            arrive(5);  // from +z
            arrive(3);  // from +y
            arrive(1);  // from +x
            rk_store<KT>(slots, w, K, sl);
            if (!tidy) occ[w] = o;
        }
        __syncthreads();
    }
}

// Pass 2 of contended frames: the serial diffusion of rdme.wgsl:45-88 in place, voxels in linear
// order.  A departing slot still holds its particle when its voxel's turn comes (arrivals only fill
// empty slots), so the snapshot has its species.  One block scans the departure bitmap; its first
// thread makes the moves.  A move changes slots, occupancy and counts alike, so a tidy voxel stays
// tidy.  Bound by one thread's dependent loads: a move reads its target's slots at once and finds the
// free one by bit tests (48 x 40 x 37, K = 8, 120,000
// particles: 70 ms per frame with a byte loop over slots, 40 now).
template <int KT>
__device__ __forceinline__ void ref_sp_serial_body(const RefParams& p, const RefSparse& sp, uint8_t* slots, uint32_t* occ,
                                                   int32_t* conc, uint32_t* diag, uint32_t* s_words) {
    const uint32_t K = KT ? (uint32_t)KT : p.K, S1 = p.S1;
    const RefMask valid = rs_valid(K);
    uint32_t spills = 0;
    for (uint32_t w0 = 0; w0 < sp.W; w0 += blockDim.x) {
        const uint32_t i = w0 + threadIdx.x;
        s_words[threadIdx.x] = i < sp.W ? ref_word(sp.dep + i) : 0u;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (uint32_t k = 0; k < blockDim.x && w0 + k < sp.W; k++) {
                uint32_t m = s_words[k];
                if (m == 0u) continue;
                const uint32_t tidy_v = sp.tidy[w0 + k];  // no pass of the moves changes it
                for (; m; m &= m - 1u) {
                    const uint32_t b = (uint32_t)(__ffs((int)m) - 1), v = (w0 + k) * 32u + b;
                    const RefSlots dr = rk_load<KT>(sp.dirs, v, K), from = rk_load<KT>(sp.snap, v, K);
                    // direction bytes below 6 (they are at most 7)
                    RefMask mv{~(dr.lo + 0x7A7A7A7A7A7A7A7Aull) & valid.lo, ~(dr.hi + 0x7A7A7A7A7A7A7A7Aull) & valid.hi};
                    for (; rm_any(mv); rm_drop(mv)) {
                        const uint32_t s = rm_first(mv), q = rs_get(from, s);
                        const uint32_t w = (uint32_t)((int64_t)v + ref_nb_offset(p, (int)rs_get(dr, s)));
                        const RefSlots to = rk_load<KT>(slots, w, K);
                        const bool tw = (sp.tidy[w >> 5] >> (w & 31u)) & 1u;
                        sp.arrivals[w] = 0u;
                        if (!tw && occ[w] >= K) { spills++; continue; }
                        const RefMask full = rs_full(to);
                        const RefMask room{~full.lo & valid.lo, ~full.hi & valid.hi};
                        if (!rm_any(room)) { spills++; continue; }
                        slots[(size_t)w * K + rm_first(room)] = (uint8_t)q;
                        slots[(size_t)v * K + s] = 0;
                        if (!tw) {
                            occ[w] += 1u;
                            conc[(size_t)w * S1 + q] = (int32_t)((uint32_t)conc[(size_t)w * S1 + q] + 1u);
                        }
                        if (!((tidy_v >> b) & 1u)) {
                            occ[v] -= 1u;
                            conc[(size_t)v * S1 + q] = (int32_t)((uint32_t)conc[(size_t)v * S1 + q] - 1u);
                        }
                    }
                }
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        diag[DIAG_SPILL] += spills;
        diag[DIAG_SLOW_STEPS] += 1u;
    }
}

// The reaction tables staged in shared memory by the reaction pass.
struct RefTables {
    const uint32_t* reactants;  // [R+1][3]
    const float* rates;         // [R+1]
    const int32_t* stoich;      // [R+1][S1]
    const uint32_t* uses;       // [S1][UW]
    const float* fire1;         // [S1]
};
__host__ __device__ constexpr size_t ref_table_words(uint32_t S1, uint32_t R, uint32_t UW) {
    return 4 * ((size_t)R + 1) + ((size_t)R + 1) * S1 + (size_t)S1 * UW + S1;
}
__device__ __forceinline__ RefTables ref_stage_tables(const RefParams& p, const RefSparse& sp, uint32_t* sm) {
    uint32_t* const s_re = sm;
    float* const s_rate = reinterpret_cast<float*>(s_re + 3 * (p.R + 1));
    int32_t* const s_st = reinterpret_cast<int32_t*>(s_rate + (p.R + 1));
    uint32_t* const s_uses = reinterpret_cast<uint32_t*>(s_st + (p.R + 1) * p.S1);
    float* const s_fire = reinterpret_cast<float*>(s_uses + p.S1 * sp.UW);
    for (uint32_t i = threadIdx.x; i < 3 * (p.R + 1); i += blockDim.x) s_re[i] = p.reactants[i];
    for (uint32_t i = threadIdx.x; i < p.R + 1; i += blockDim.x) s_rate[i] = p.rates[i];
    for (uint32_t i = threadIdx.x; i < (p.R + 1) * p.S1; i += blockDim.x) s_st[i] = p.stoich[i];
    for (uint32_t i = threadIdx.x; i < p.S1 * sp.UW; i += blockDim.x) s_uses[i] = sp.uses[i];
    for (uint32_t i = threadIdx.x; i < p.S1; i += blockDim.x) s_fire[i] = sp.fire1[i];
    return RefTables{s_re, s_rate, s_st, s_uses, s_fire};
}

// The reaction pass on voxel v (tidy or not), as ref_cme_voxel; `row` is the thread's shared-memory
// concentration row.  Returns whether the voxel stays in act; `tidy` as it is afterwards.
template <int KT>
__device__ __forceinline__ bool ref_react(const RefParams& p, const RefSparse& sp, const RefTables& T, uint32_t v,
                                          uint8_t* slots, uint32_t* occ, int32_t* conc, uint32_t itime,
                                          int32_t* s_delta, int32_t* row, bool& tidy) {
    const uint32_t K = KT ? (uint32_t)KT : p.K, S1 = p.S1, R = p.R, S = S1 - 1u;
    const RefSlots snap = rk_load<KT>(slots, v, K);
    uint32_t x, y, z;
    ref_coords(p, v, x, y, z);
    const uint32_t state = d_pcg(itime + x * y + z);
    const float r1 = d_uniform_float(state);
    RefMask full = rs_full(snap);
    const uint32_t n = rm_count(full);
    const bool was = tidy;
    RefSlots sl = snap;
    bool fires;
    bool have_row = false;
    int32_t* const c = conc + (size_t)v * S1;
    auto make_row = [&]() {
        have_row = true;
        if (was) {
            row[0] = 1;
            for (uint32_t s = 1; s < S1; s++) row[s] = 0;
            for (RefMask f = full; rm_any(f); rm_drop(f)) row[rs_get(snap, rm_first(f))]++;
        } else {
            for (uint32_t s = 0; s < S1; s++) row[s] = c[s];
            if (row[0] != 1) {
                row[0] = 1;
                c[0] = 1;
            }
        }
    };
    auto prop_of = [&](uint32_t r) -> float {
        const uint32_t prod = (uint32_t)row[T.reactants[r * 3]] * (uint32_t)row[T.reactants[r * 3 + 1]] *
                              (uint32_t)row[T.reactants[r * 3 + 2]];
        return __fmul_rn(T.rates[r], __int2float_rn((int32_t)prod));
    };
    float total = 0.0f;
    auto sum = [&]() {
        total = 0.0f;
        if (sp.finite) {  // a reaction that lacks a reactant adds a zero, which changes no sum
            for (uint32_t u = 0; u < sp.UW; u++) {
                uint32_t m = 0xFFFFFFFFu;
                for (uint32_t s = 1; s < S1; s++)
                    if (row[s] == 0) m &= ~T.uses[s * sp.UW + u];
                if (u == 0u) m &= ~1u;
                if (32u * u + 31u > R) m &= R >= 32u * u ? (2u << (R - 32u * u)) - 1u : 0u;
                for (; m; m &= m - 1u) total = __fadd_rn(total, prop_of(32u * u + (uint32_t)(__ffs((int)m) - 1)));
            }
        } else {
            for (uint32_t r = 1; r <= R; r++) total = __fadd_rn(total, prop_of(r));
        }
    };
    if (was && n <= 1u) {
        fires = r1 <= T.fire1[n ? rs_get(snap, rm_first(full)) : 0u];
    } else {
        make_row();
        sum();
        fires = r1 <= __fsub_rn(1.0f, d_expf(__fmul_rn(-total, p.tau)));
    }
    if (fires) {
        if (!have_row) {
            make_row();
            sum();
        }
        atomicAdd(&s_delta[S1], 1);
        const float r2 = d_uniform_float(state + 1u);
        // selection over cum[i] = cum[i-1] + a_i, normalised for i < R (cme.wgsl:50-52,70-73)
        uint32_t i = 0;
        float run = 0.0f;
        while (i < R) {
            if (!(r2 > __fdiv_rn(run, total))) break;
            i++;
            run = __fadd_rn(run, prop_of(i));
        }
        const int32_t* st = T.stoich + (size_t)i * S1;
        uint32_t j = 0;
        const int32_t occ0 = was ? (int32_t)n : (int32_t)occ[v];
        int32_t new_occ = occ0;
        const uint64_t ri = (uint64_t)v * K;  // reservoirs[idx_lattice], cme.wgsl:80
        const uint32_t resv = (ri < p.V) ? p.reservoir[ri] : 0u;
        bool rolled = false;
        for (uint32_t s = 1; s <= S && !rolled; s++) {
            if (resv == s) continue;
            const int32_t d = st[s];
            row[s] = (int32_t)((uint32_t)row[s] + (uint32_t)d);
            new_occ = (int32_t)((uint32_t)new_occ + (uint32_t)d);
            if (d) atomicAdd(&s_delta[s], d);
            int32_t cc = row[s];
            while (cc > 0) {
                rs_set(sl, j, s);
                cc--;
                j++;
                if (j >= K) {
                    sl = snap;
                    for (uint32_t s2 = 1; s2 <= s; s2++) {
                        const int32_t d2 = st[s2];
                        row[s2] = (int32_t)((uint32_t)row[s2] - (uint32_t)d2);
                        if (d2) atomicAdd(&s_delta[s2], -d2);
                    }
                    atomicAdd(&s_delta[S1 + 1], 1);
                    rolled = true;
                    break;
                }
            }
        }
        if (!rolled) {
            while (j < K) rs_set(sl, j++, 0u);
        } else {
            new_occ = occ0;
        }
        // do the new slots still imply the occupancy and the counts?
        const RefMask f1 = rs_full(sl);
        bool same = new_occ == (int32_t)rm_count(f1);
        for (RefMask f = f1; rm_any(f); rm_drop(f)) row[rs_get(sl, rm_first(f))]--;
        for (uint32_t s = 1; s < S1; s++) same &= row[s] == 0;
        for (RefMask f = f1; rm_any(f); rm_drop(f)) row[rs_get(sl, rm_first(f))]++;
        tidy = same;
        if (!same) {
            for (uint32_t s = 0; s < S1; s++) c[s] = row[s];
            occ[v] = (uint32_t)new_occ;
        }
        full = f1;
    }
    // stable move of the non-zero slots to the front
    auto packed = [](uint64_t f) -> bool {  // bytes marked from the lowest on
        const uint64_t t = f | (f - (f >> 7));
        return (t & (t + 1ull)) == 0ull;
    };
    RefSlots out = sl;
    if (!(packed(full.lo) && packed(full.hi) && (full.hi == 0ull || full.lo == 0x8080808080808080ull))) {
        out = RefSlots{0ull, 0ull};
        uint32_t jj = 0;
        for (RefMask f = full; rm_any(f); rm_drop(f)) rs_set(out, jj++, rs_get(sl, rm_first(f)));
    }
    if (out.lo != snap.lo || out.hi != snap.hi) rk_store<KT>(slots, v, K, out);
    bool keep = rm_any(full);
    if (!tidy && !keep) {
        keep = occ[v] != 0u;
        for (uint32_t s = 1; s < S1 && !keep; s++) keep |= row[s] != 0;
    }
    return keep;
}

// Pass 3: the reaction pass over act and touch (every voxel when `dense`), which leaves the next
// frame's act words and clears the touch and departure words.  rows: the staged tables and a
// shared-memory row per thread are used (else, when they do not fit, the global-memory form; no
// voxel is tidy then).
template <int KT, int NT>
__device__ __forceinline__ void ref_sp_cme_body(const RefParams& p, const RefSparse& sp, uint8_t* slots, uint32_t* occ,
                                                int32_t* conc, uint32_t itime, uint32_t dense, const RefRange& R,
                                                const RefTables& T, int32_t* s_delta, int32_t* row, uint32_t rows) {
    const uint32_t K = KT ? (uint32_t)KT : p.K;
    for (uint32_t w0 = blockIdx.x * sp.cw; w0 < sp.W; w0 += gridDim.x * sp.cw) {
        const uint32_t i = w0 + threadIdx.x;
        const bool own = threadIdx.x < sp.cw && i < sp.W;
        uint32_t m = 0u, a = 0u, t = 0u, tidy0 = 0u;
        if (own) {
            a = sp.act[i];
            t = ref_word(sp.touch + i);
            tidy0 = sp.tidy[i];
            m = a | t;
            if (dense) m = (uint64_t)i * 32u + 32u <= p.V ? 0xFFFFFFFFu : (1u << (p.V & 31u)) - 1u;
            R.area[RW_A][threadIdx.x] = tidy0;
            R.area[RW_B][threadIdx.x] = 0u;   // the next act word
            R.area[RW_C][threadIdx.x] = tidy0;  // the next tidy word
        }
        const uint32_t n = ref_list<NT>(m, R);
        for (uint32_t e = threadIdx.x; e < n; e += NT) {
            const uint32_t idx = R.list[e] >> 5, b = R.list[e] & 31u, bit = 1u << b;
            const uint32_t v = (w0 + idx) * 32u + b;
            bool keep;
            if (rows) {
                const bool was = R.area[RW_A][idx] & bit;
                bool tidy = was;
                keep = ref_react<KT>(p, sp, T, v, slots, occ, conc, itime, s_delta, row, tidy);
                if (tidy != was) atomicXor(&R.area[RW_C][idx], bit);
            } else {
                ref_cme_voxel(p, v, slots, occ, conc, itime, s_delta);
                keep = occ[v] != 0u || rm_any(rs_full(rk_load<KT>(slots, v, K)));
                for (uint32_t s = 1; s < p.S1 && !keep; s++) keep |= conc[(size_t)v * p.S1 + s] != 0;
            }
            if (keep) atomicOr(&R.area[RW_B][idx], bit);
        }
        __syncthreads();
        if (own) {
            const uint32_t keep = R.area[RW_B][threadIdx.x], tidy = R.area[RW_C][threadIdx.x];
            if (keep != a) sp.act[i] = keep;
            if (tidy != tidy0) sp.tidy[i] = tidy;
            if (t) {
                sp.touch[i] = 0u;
                sp.dep[i] = 0u;  // a voxel with a departure is touched
            }
        }
        __syncthreads();
    }
}

// Threads of a block of the three launches.
constexpr int REF_NT = 128;
constexpr size_t REF_SMEM = 44u * 1024u;  // dynamic shared memory of a launch without an attribute, and some for static

template <int KT>
__global__ void __launch_bounds__(REF_NT) ref_sp_directions(const __grid_constant__ RefParams p,
                                                            const __grid_constant__ RefSparse sp, const uint8_t* slots,
                                                            const uint32_t* occ, const uint32_t* itimes, uint32_t step,
                                                            uint32_t* diag, uint32_t* contended, uint32_t stage_P) {
    extern __shared__ __align__(16) uint32_t sm[];
    float* const s_P = reinterpret_cast<float*>(sm + ref_range_words(sp.cw));
    ref_allow_next();
    ref_stage_P(p, s_P, stage_P);
    const uint32_t itime = __ldg(itimes + step);
    ref_wait_previous();
    ref_sp_directions_body<KT, REF_NT>(p, sp, slots, occ, itime, diag, contended, ref_range(sm, sp.cw), stage_P ? s_P : p.P);
}

template <int KT>
__global__ void __launch_bounds__(REF_NT) ref_sp_move(const __grid_constant__ RefParams p,
                                                      const __grid_constant__ RefSparse sp, uint8_t* slots, uint32_t* occ,
                                                      int32_t* conc, uint32_t* diag, const uint32_t* contended) {
    extern __shared__ __align__(16) uint32_t sm[];
    ref_allow_next();
    ref_wait_previous();
    if (ref_word(contended)) {
        if (blockIdx.x == 0) {
            __shared__ uint32_t s_words[REF_NT];
            ref_sp_serial_body<KT>(p, sp, slots, occ, conc, diag, s_words);
        }
        return;
    }
    ref_sp_gather_body<KT, REF_NT>(p, sp, slots, occ, conc, ref_range(sm, sp.cw));
}

// Shared memory of the reaction pass behind the range: S1 + 2 counters, then (rows) the tables and rows.
template <int KT>
__global__ void __launch_bounds__(REF_NT) ref_sp_cme(const __grid_constant__ RefParams p,
                                                     const __grid_constant__ RefSparse sp, uint8_t* slots, uint32_t* occ,
                                                     int32_t* conc, const uint32_t* itimes, uint32_t step, uint32_t dense,
                                                     int32_t* stat, uint32_t* diag, uint32_t* contended, uint32_t rows) {
    extern __shared__ __align__(16) uint32_t sm[];
    int32_t* const s_delta = reinterpret_cast<int32_t*>(sm + ref_range_words(sp.cw));
    ref_allow_next();
    for (uint32_t s = threadIdx.x; s < p.S1 + 2; s += REF_NT) s_delta[s] = 0;
    uint32_t* const s_tab = reinterpret_cast<uint32_t*>(s_delta + p.S1 + 2);
    RefTables T{};
    if (rows) T = ref_stage_tables(p, sp, s_tab);
    int32_t* const row = reinterpret_cast<int32_t*>(s_tab + ref_table_words(p.S1, p.R, sp.UW)) + threadIdx.x * p.S1;
    const uint32_t itime = __ldg(itimes + step);
    ref_wait_previous();
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) *contended = 0u;  // every reader of this frame's flag has run
    ref_sp_cme_body<KT, REF_NT>(p, sp, slots, occ, conc, itime, dense, ref_range(sm, sp.cw), T, s_delta, row, rows);
    ref_flush_block(p, s_delta, stat, diag);
}

// Threads of the one-block form below.
constexpr int REF_BLOCK_THREADS = 512;
// Lattices of at most this many voxels and (when they are uploaded) particles run every frame of a call
// in the one-block form, if its state and a row per thread fit in shared memory.  us per frame, one block
// / three launches: 64 x 64 x 1, K = 8, with 200 particles 9.0 / 12.9, 400 10.0 / 13.5, 800 15.2 / 14.5; 77 x
// 78 x 1 with 600 13.3 / 13.9, 1,100 19.0 / 14.6; without the rows, 16^3, K = 16, 300 particles 27 / 13.4.  The
// block's time is one SM's dependent steps (about a dozen barriers and the entries' instruction chains) and
// follows the particles; the launches' is three launch latencies whatever the size up to about 40^3.  With
// the state in global memory the block took 12.4 at 400 particles: a frame was a chain of L2 round trips.
constexpr uint64_t REF_BLOCK_MAX_VOXELS = 6144, REF_BLOCK_MAX_PARTICLES = 600;

// Every frame of a step call in one block: the passes' own bodies in the same order, with block
// barriers where the launches were (the serial pass runs on the same block).  What the frames read and
// write (slots, bitmaps, arrivals, directions and snapshots) is in shared memory for the whole call;
// the occupancy and rows of voxels that are not tidy stay in global memory, and the bodies read
// nothing that the block writes through the non-coherent path.
template <int KT>
__global__ void __launch_bounds__(REF_BLOCK_THREADS, 1)
    ref_sp_frames_block(const __grid_constant__ RefParams p, const __grid_constant__ RefSparse g, uint8_t* g_slots,
                        uint32_t* occ, int32_t* conc, const uint32_t* itimes, uint32_t step0, uint32_t n,
                        uint32_t dense_first, uint32_t dense_always, int32_t* stat, uint32_t* diag,
                        uint32_t* g_contended, uint32_t stage_P, uint32_t rows, uint32_t other) {
    constexpr int NT = REF_BLOCK_THREADS;
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ uint32_t s_words[NT];
    __shared__ uint32_t s_contended;
    uint32_t* const contended = &s_contended;
    // the state, behind `other` bytes of lists and tables
    RefSparse sp = g;
    const uint32_t V = (uint32_t)p.V, VK = (uint32_t)(p.V * p.K), VKa = (VK + 15u) & ~15u;
    uint8_t* const s_state = reinterpret_cast<uint8_t*>(sm) + other;
    uint8_t* const slots = s_state;
    sp.dirs = slots + VKa;
    sp.snap = sp.dirs + VKa;
    sp.arrivals = reinterpret_cast<uint32_t*>(sp.snap + VKa);
    sp.act = sp.arrivals + V;
    sp.touch = sp.act + g.W;
    sp.dep = sp.touch + g.W;
    sp.tidy = sp.dep + g.W;
    for (uint32_t i = threadIdx.x; i < VKa / 4u; i += NT)
        if (4u * i + 4u <= VK) reinterpret_cast<uint32_t*>(slots)[i] = reinterpret_cast<const uint32_t*>(g_slots)[i];
    for (uint32_t i = threadIdx.x; i < V; i += NT) sp.arrivals[i] = 0u;
    for (uint32_t i = threadIdx.x; i < g.W; i += NT) {
        sp.act[i] = g.act[i];
        sp.touch[i] = sp.dep[i] = 0u;
        sp.tidy[i] = g.tidy[i];
    }
    if (threadIdx.x == 0) {
        *contended = *g_contended;
        for (uint32_t i = VK & ~3u; i < VK; i++) slots[i] = g_slots[i];  // a last, partial word
    }
    const RefRange R = ref_range(sm, sp.cw);
    int32_t* const s_delta = reinterpret_cast<int32_t*>(sm + ref_range_words(sp.cw));
    float* const s_P = reinterpret_cast<float*>(s_delta + p.S1 + 2);
    uint32_t* const s_tab = reinterpret_cast<uint32_t*>(s_P + (stage_P ? p.NR * p.NR * p.S1 : 0u));
    ref_stage_P(p, s_P, stage_P);
    for (uint32_t s = threadIdx.x; s < p.S1 + 2; s += NT) s_delta[s] = 0;
    RefTables T{};
    if (rows) T = ref_stage_tables(p, sp, s_tab);
    int32_t* const row = reinterpret_cast<int32_t*>(s_tab + ref_table_words(p.S1, p.R, sp.UW)) + threadIdx.x * p.S1;
    __syncthreads();
    for (uint32_t k = 0; k < n; k++) {
        const uint32_t itime = __ldg(itimes + step0 + k);
        ref_sp_directions_body<KT, NT>(p, sp, slots, occ, itime, diag, contended, R, stage_P ? s_P : p.P);
        __syncthreads();
        const uint32_t full = ref_word(contended);
        if (full) ref_sp_serial_body<KT>(p, sp, slots, occ, conc, diag, s_words);
        else ref_sp_gather_body<KT, NT>(p, sp, slots, occ, conc, R);
        __syncthreads();
        if (full && threadIdx.x == 0) *contended = 0u;  // every thread has read it
        const uint32_t dense = ((k == 0u && dense_first) || dense_always) ? 1u : 0u;
        ref_sp_cme_body<KT, NT>(p, sp, slots, occ, conc, itime, dense, R, T, s_delta, row, rows);
        __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < VK / 4u; i += NT)
        reinterpret_cast<uint32_t*>(g_slots)[i] = reinterpret_cast<const uint32_t*>(slots)[i];
    for (uint32_t i = (VK & ~3u) + threadIdx.x; i < VK; i += NT) g_slots[i] = slots[i];
    for (uint32_t i = threadIdx.x; i < g.W; i += NT) {
        g.act[i] = sp.act[i];
        g.tidy[i] = sp.tidy[i];
    }
    if (threadIdx.x == 0) *g_contended = 0u;
    ref_flush_block(p, s_delta, stat, diag);
}

// act and tidy of a freshly uploaded lattice, a warp per word (no voxel is tidy without `rows`).
__global__ void __launch_bounds__(256) ref_sp_build(RefParams p, RefSparse sp, const uint8_t* slots, const uint32_t* occ,
                                                    const int32_t* conc, uint32_t rows) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t i = blockIdx.x * 8u + (threadIdx.x >> 5); i < sp.W; i += gridDim.x * 8u) {
        const uint64_t v = (uint64_t)i * 32u + lane;
        bool keep = false, tidy = false;
        if (v < p.V) {
            const RefSlots sl = rs_load(slots + v * p.K, p.K);
            const RefMask full = rs_full(sl);
            tidy = rows != 0u && occ[v] == rm_count(full);
            keep = occ[v] != 0u || rm_any(full);
            for (uint32_t s = 1; s < p.S1; s++) {
                int32_t n = 0;
                for (RefMask f = full; rm_any(f); rm_drop(f)) n += rs_get(sl, rm_first(f)) == s;
                const int32_t c = conc[v * p.S1 + s];
                keep |= c != 0;
                tidy &= c == n;
            }
            for (RefMask f = full; rm_any(f); rm_drop(f)) tidy &= rs_get(sl, rm_first(f)) < p.S1;
        }
        const uint32_t k = __ballot_sync(0xffffffffu, keep), t = __ballot_sync(0xffffffffu, tidy);
        if (lane == 0u) {
            sp.act[i] = k;
            sp.tidy[i] = t;
        }
    }
}

// The occupancy and the concentration rows of the tidy voxels, from their slots (frames have run: their
// first reaction pass has set every row's entry 0).
__global__ void __launch_bounds__(256) ref_write_rows(RefParams p, RefSparse sp, const uint8_t* slots, uint32_t* occ,
                                                      int32_t* conc) {
    for (uint64_t v = (uint64_t)blockIdx.x * 256u + threadIdx.x; v < p.V; v += (uint64_t)gridDim.x * 256u) {
        if (!bit_of(sp.tidy, (uint32_t)v)) continue;
        const RefSlots sl = rs_load(slots + v * p.K, p.K);
        RefMask full = rs_full(sl);
        int32_t* const c = conc + v * p.S1;
        occ[v] = rm_count(full);
        c[0] = 1;
        for (uint32_t s = 1; s < p.S1; s++) c[s] = 0;
        for (; rm_any(full); rm_drop(full)) c[rs_get(sl, rm_first(full))]++;
    }
}

// Voxels whose six neighbours lie in the lattice and share their region, a warp per word.
__global__ void __launch_bounds__(256) ref_same_regions(RefParams p, uint32_t* same, uint32_t W) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t i = blockIdx.x * 8u + (threadIdx.x >> 5); i < W; i += gridDim.x * 8u) {
        const uint64_t v = (uint64_t)i * 32u + lane;
        bool is = false;
        if (v < p.V) {
            uint32_t x, y, z;
            ref_coords(p, (uint32_t)v, x, y, z);
            if (x > 0u && x < p.X - 1u && y > 0u && y < p.Y - 1u && z > 0u && z < p.Z - 1u) {
                const uint8_t* r = p.regions + v;
                const uint8_t q = *r;
                is = r[-(int64_t)p.YZ] == q && r[p.YZ] == q && r[-(int64_t)p.Z] == q && r[p.Z] == q && r[-1] == q && r[1] == q;
            }
        }
        const uint32_t m = __ballot_sync(0xffffffffu, is);
        if (lane == 0u) same[i] = m;
    }
}

// RefSparse::fire1: the propensity sum of a voxel whose only particle is q, by the operations of the
// reaction pass in their order.
__global__ void ref_fire_table(RefParams p, float* fire1) {
    for (uint32_t q = threadIdx.x; q < p.S1; q += blockDim.x) {
        float total = 0.0f;
        for (uint32_t r = 1; r <= p.R; r++) {
            uint32_t prod = 1u;
            for (uint32_t j = 0; j < 3; j++) {
                const uint32_t a = p.reactants[r * 3 + j];
                prod *= (a == 0u || a == q) ? 1u : 0u;
            }
            total = __fadd_rn(total, __fmul_rn(p.rates[r], __int2float_rn((int32_t)prod)));
        }
        fire1[q] = __fsub_rn(1.0f, d_expf(__fmul_rn(-total, p.tau)));
    }
}

// ------------------------------------------------------------------ host side

// Bytes of the one-block form's state.
static size_t ref_state_bytes(const RefParams& p) {
    const size_t VKa = ((size_t)(p.V * p.K) + 15u) & ~(size_t)15u, W = ((size_t)p.V + 31u) / 32u;
    return 3 * VKa + 4 * (size_t)p.V + 16 * W;
}
static bool ref_one_block(const DeviceRef* d) { return d->one_block; }

static RefSparse ref_sparse(DeviceRef* d) {
    RefSparse sp{};
    sp.act = d->act_bm.p;
    sp.touch = d->touch_bm.p;
    sp.dep = d->dep_bm.p;
    sp.tidy = d->tidy_bm.p;
    sp.same = d->same_bm.p;
    sp.arrivals = d->arrivals.p;
    sp.dirs = d->dirs.p;
    sp.snap = d->snap.p;
    sp.uses = d->uses.p;
    sp.fire1 = d->fire1.p;
    sp.W = (uint32_t)d->touch_bm.n;
    // a range per block: four blocks per SM where the lattice has the words for it (us per frame with two /
    // four / eight: 64^3 with 22,000 particles 19.7 / 18.5 / 21.9, 100^3 with 40,000 29.9 / 24.2 / 29.3), and no
    // more words than a block has threads
    sp.cw = ref_one_block(d) ? sp.W : std::min<uint32_t>(REF_NT, std::max<uint32_t>(1u, sp.W / (4u * (uint32_t)d->sms)));
    sp.UW = d->p.R / 32u + 1u;
    sp.finite = d->finite ? 1u : 0u;
    return sp;
}

// Shared memory (bytes) of the passes in blocks of nt threads, with ranges of cw words: the range, the
// S1 + 2 counters and, when they fit beside them in `limit` (rows), the reaction tables and a row per
// thread; the directions pass stages the probability table when it takes at most 16 KB.
static size_t ref_cme_smem(const RefParams& p, const RefSparse& sp, int nt, size_t other, size_t limit, uint32_t& rows) {
    const size_t base = (ref_range_words(sp.cw) + p.S1 + 2) * 4 + other;
    const size_t all = base + (ref_table_words(p.S1, p.R, sp.UW) + (size_t)nt * p.S1) * 4;
    rows = all <= limit ? 1u : 0u;
    return rows ? all : base;
}
static size_t ref_P_smem(const RefParams& p, uint32_t& stage_P) {
    const size_t smem_P = (size_t)p.NR * p.NR * p.S1 * sizeof(float);
    stage_P = smem_P <= 16u * 1024u ? 1u : 0u;
    return stage_P ? smem_P : 0u;
}

// Shared memory of the one-block form, or 0 when it does not fit; other: the bytes before its state.
static size_t ref_block_smem(const DeviceRef* d, const RefSparse& sp, uint32_t& stage_P, uint32_t& rows, uint32_t& other) {
    const size_t P = ref_P_smem(d->p, stage_P);
    const size_t state = ref_state_bytes(d->p) + 16u, most = (size_t)d->smem_optin - 4096u;
    if (state >= most) return 0u;
    other = (uint32_t)((ref_cme_smem(d->p, sp, REF_BLOCK_THREADS, P, most - state, rows) + 15u) & ~(size_t)15u);
    const size_t all = other + state;
    return all <= most ? all : 0u;
}

// Whether the reaction pass runs on shared-memory rows (tidy voxels need them).
static uint32_t ref_rows(const DeviceRef* d, const RefSparse& sp) {
    uint32_t rows = 0, stage_P = 0, other = 0;
    if (ref_one_block(d)) ref_block_smem(d, sp, stage_P, rows, other);
    else ref_cme_smem(d->p, sp, REF_NT, 0, REF_SMEM, rows);
    return rows;
}

template <int KT>
static void ref_block_attr(int bytes) {
    CS_CUDA(cudaFuncSetAttribute(ref_sp_frames_block<KT>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

// Chooses the form for a lattice of `particles` particles.
static void ref_choose_form(DeviceRef* d, uint64_t particles) {
    d->one_block = d->p.V <= REF_BLOCK_MAX_VOXELS && particles <= REF_BLOCK_MAX_PARTICLES;
    if (!d->one_block) return;
    uint32_t rows = 0, stage_P = 0, other = 0;
    if (!ref_block_smem(d, ref_sparse(d), stage_P, rows, other) || !rows) {
        d->one_block = false;
        return;
    }
    const int most = d->smem_optin - 4096;
    if (d->p.K == 16u) ref_block_attr<16>(most);
    else if (d->p.K == 8u) ref_block_attr<8>(most);
    else ref_block_attr<0>(most);
}

static void ref_bind(DeviceRef* d) {
    d->p.P = d->P.p;
    d->p.stoich = d->stoich.p;
    d->p.reactants = d->reactants.p;
    d->p.rates = d->rates.p;
    d->p.regions = d->regions.p;
    d->p.reservoir = d->reservoir.p;
}

DeviceRef* ref_create(const Model& m, int device) {
    m.check_tables();
    if (m.n_reactions > 99) throw Error(CS_ERR_LIMIT, "at most 99 reactions");
    if (m.V * m.K >= (1ull << 32))
        throw Error(CS_ERR_LIMIT, "the reference-RNG path indexes slots with u32: V * K must be below 2^32");
    if (m.nr > 256) throw Error(CS_ERR_LIMIT, "at most 256 regions");
    if (m.n_species > 255) throw Error(CS_ERR_LIMIT, "at most 255 species");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
        throw Error(CS_ERR_CUDA, "no CUDA device available (libcellsim has no CPU fallback)");
    if (device < 0 || device >= ndev) throw Error(CS_ERR_INVALID_ARG, "device index out of range");
    DeviceGuard g(device);
    std::unique_ptr<DeviceRef> d(new DeviceRef());
    d->device = device;
    CS_CUDA(cudaStreamCreateWithFlags(&d->stream, cudaStreamNonBlocking));
    RefParams& p = d->p;
    p.X = m.res[0]; p.Y = m.res[1]; p.Z = m.res[2];
    p.K = m.K; p.S1 = m.n_species + 1; p.R = m.n_reactions; p.NR = m.nr;
    p.YZ = p.Y * p.Z;
    p.V = m.V;
    p.tau = m.tau;
    uint64_t VK = m.V * m.K, VS = m.V * p.S1;
    d->slots.alloc(VK);
    d->occ.alloc(m.V);
    d->conc.alloc(VS);
    d->regions.alloc(m.V);
    d->reservoir.alloc(m.V);
    d->dirs.alloc(VK);
    d->snap.alloc(VK);
    const uint64_t W = (m.V + 31) / 32;
    d->act_bm.alloc(W);
    d->touch_bm.alloc(W);
    d->dep_bm.alloc(W);
    d->tidy_bm.alloc(W);
    d->same_bm.alloc(W);
    d->arrivals.alloc(m.V);
    CS_CUDA(cudaMemset(d->arrivals.p, 0, m.V * 4));
    CS_CUDA(cudaDeviceGetAttribute(&d->sms, cudaDevAttrMultiProcessorCount, device));
    CS_CUDA(cudaDeviceGetAttribute(&d->smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    for (uint32_t r = 1; r <= m.n_reactions; r++)
        if (m.reactants[r * 3] == 0u && m.reactants[r * 3 + 1] == 0u && m.reactants[r * 3 + 2] == 0u)
            d->dense_always = true;
    std::vector<float> P;
    compute_ref_probabilities(m, P);
    d->P.alloc(P.size());
    d->rates.alloc(m.rates.size());
    d->stoich.alloc(m.stoich.size());
    d->reactants.alloc(m.reactants.size());
    d->stat.alloc(p.S1);
    d->diag.alloc(DIAG_N);
    d->flag.alloc(1);
    ref_bind(d.get());
    std::vector<uint8_t> r8(m.V), res8(m.V);
    for (uint64_t v = 0; v < m.V; v++) { r8[v] = (uint8_t)m.regions[v]; res8[v] = (uint8_t)m.reservoir[v]; }
    CS_CUDA(cudaMemcpy(d->regions.p, r8.data(), m.V, cudaMemcpyHostToDevice));
    CS_CUDA(cudaMemcpy(d->reservoir.p, res8.data(), m.V, cudaMemcpyHostToDevice));
    CS_CUDA(cudaMemcpy(d->P.p, P.data(), P.size() * sizeof(float), cudaMemcpyHostToDevice));
    CS_CUDA(cudaMemcpy(d->rates.p, m.rates.data(), m.rates.size() * sizeof(float), cudaMemcpyHostToDevice));
    CS_CUDA(cudaMemcpy(d->stoich.p, m.stoich.data(), m.stoich.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
    CS_CUDA(cudaMemcpy(d->reactants.p, m.reactants.data(), m.reactants.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    CS_CUDA(cudaMemset(d->diag.p, 0, DIAG_N * sizeof(uint32_t)));
    CS_CUDA(cudaMemset(d->flag.p, 0, sizeof(uint32_t)));
    const uint32_t UW = p.R / 32u + 1u;
    std::vector<uint32_t> uses((size_t)p.S1 * UW, 0u);
    for (uint32_t r = 1; r <= p.R; r++) {
        d->finite = d->finite && std::isfinite(m.rates[r]);
        for (uint32_t j = 0; j < 3; j++) uses[(size_t)m.reactants[r * 3 + j] * UW + r / 32u] |= 1u << (r & 31u);
    }
    d->uses.alloc(uses.size());
    CS_CUDA(cudaMemcpy(d->uses.p, uses.data(), uses.size() * 4, cudaMemcpyHostToDevice));
    d->fire1.alloc(p.S1);
    ref_fire_table<<<1, 256, 0, d->stream>>>(p, d->fire1.p);
    CS_LAUNCH_CHECK();
    ref_same_regions<<<2048, 256, 0, d->stream>>>(p, d->same_bm.p, (uint32_t)W);
    CS_LAUNCH_CHECK();
    std::vector<int32_t> conc = m.concentrations();
    ref_set_lattice(d.get(), m.slots.data(), m.occupancy.data(), conc.data());
    return d.release();
}

void ref_destroy(DeviceRef* d) {
    if (!d) return;
    cudaSetDevice(d->device);
    if (d->stream) cudaStreamSynchronize(d->stream);
    delete d;
}

void ref_set_lattice(DeviceRef* d, const uint32_t* slots, const uint32_t* occ, const int32_t* conc) {
    DeviceGuard g(d->device);
    uint64_t VK = d->p.V * d->p.K, VS = d->p.V * d->p.S1;
    std::vector<uint8_t> s8(VK);
    for (uint64_t i = 0; i < VK; i++) {
        if (slots[i] > 255u) throw Error(CS_ERR_LIMIT, "slot value above 255");
        s8[i] = (uint8_t)slots[i];
    }
    CS_CUDA(cudaStreamSynchronize(d->stream));
    CS_CUDA(cudaMemcpy(d->slots.p, s8.data(), VK, cudaMemcpyHostToDevice));
    CS_CUDA(cudaMemcpy(d->occ.p, occ, d->p.V * sizeof(uint32_t), cudaMemcpyHostToDevice));
    CS_CUDA(cudaMemcpy(d->conc.p, conc, VS * sizeof(int32_t), cudaMemcpyHostToDevice));
    // the sparse passes start from the act bitmap of the new lattice and empty touch and departure
    // bitmaps; its first reaction pass visits every voxel (conc[v][0] = 1, compaction)
    const size_t wb = d->touch_bm.bytes();
    CS_CUDA(cudaMemset(d->touch_bm.p, 0, wb));
    CS_CUDA(cudaMemset(d->dep_bm.p, 0, wb));
    CS_CUDA(cudaMemset(d->arrivals.p, 0, d->arrivals.bytes()));
    uint64_t particles = 0;
    for (uint64_t i = 0; i < VK; i++) particles += s8[i] != 0u;
    ref_choose_form(d, particles);
    const RefSparse sp = ref_sparse(d);
    ref_sp_build<<<d->sms * 8, 256, 0, d->stream>>>(d->p, sp, d->slots.p, d->occ.p, d->conc.p, ref_rows(d, sp));
    CS_LAUNCH_CHECK();
    d->rows_stale = false;
    CS_CUDA(cudaStreamSynchronize(d->stream));
    d->dense_next = true;
    // create_statistics, src/simulation.rs:361-388: the counts restart from the sum of the concentrations
    std::vector<int32_t> st(d->p.S1, 0);
    for (uint64_t v = 0; v < d->p.V; v++)
        for (uint32_t s = 0; s < d->p.S1; s++) st[s] = (int32_t)((uint32_t)st[s] + (uint32_t)conc[v * d->p.S1 + s]);
    CS_CUDA(cudaMemcpy(d->stat.p, st.data(), d->p.S1 * sizeof(int32_t), cudaMemcpyHostToDevice));
}

void ref_set_counts(DeviceRef* d, const int64_t* counts) {
    DeviceGuard g(d->device);
    std::vector<int32_t> st(d->p.S1);
    for (uint32_t s = 0; s < d->p.S1; s++) st[s] = (int32_t)counts[s];
    CS_CUDA(cudaStreamSynchronize(d->stream));
    CS_CUDA(cudaMemcpy(d->stat.p, st.data(), d->p.S1 * sizeof(int32_t), cudaMemcpyHostToDevice));
}

void ref_render_view(DeviceRef* d, int32_t view, int32_t slice_axis, uint32_t slice, float* out_host, void* out_device) {
    DeviceGuard g(d->device);
    DevBuf<float> tmp;
    float* out_dev = static_cast<float*>(out_device);
    if (!out_dev) {
        tmp.alloc(d->p.V);
        out_dev = tmp.p;
    }
    ViewParams v{};
    v.slots = d->slots.p;
    v.K = d->p.K;
    v.X = d->p.X; v.Y = d->p.Y; v.Z = d->p.Z;
    v.region_id = d->regions.p;
    v.reservoir = d->reservoir.p;
    v.view = view;
    v.slice_axis = slice_axis;
    v.slice = slice;
    v.out = out_dev;
    if (view == 0 && slice == 0u && (v.K == 8u || v.K == 16u)) launch_majority_view(v.K, v.slots, d->p.V, out_dev, d->stream);
    else render_view_kernel<<<1024, 256, 0, d->stream>>>(v);
    CS_LAUNCH_CHECK();
    if (!out_device) CS_CUDA(cudaMemcpyAsync(out_host, out_dev, d->p.V * sizeof(float), cudaMemcpyDeviceToHost, d->stream));
    CS_CUDA(cudaStreamSynchronize(d->stream));
}

void ref_get_lattice(DeviceRef* d, uint32_t* slots, uint32_t* occ, int32_t* conc) {
    DeviceGuard g(d->device);
    if ((occ || conc) && d->rows_stale) {
        ref_write_rows<<<d->sms * 8, 256, 0, d->stream>>>(d->p, ref_sparse(d), d->slots.p, d->occ.p, d->conc.p);
        CS_LAUNCH_CHECK();
        d->rows_stale = false;
    }
    CS_CUDA(cudaStreamSynchronize(d->stream));
    uint64_t VK = d->p.V * d->p.K, VS = d->p.V * d->p.S1;
    if (slots) {
        std::vector<uint8_t> s8(VK);
        CS_CUDA(cudaMemcpy(s8.data(), d->slots.p, VK, cudaMemcpyDeviceToHost));
        for (uint64_t i = 0; i < VK; i++) slots[i] = s8[i];
    }
    if (occ) CS_CUDA(cudaMemcpy(occ, d->occ.p, d->p.V * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    if (conc) CS_CUDA(cudaMemcpy(conc, d->conc.p, VS * sizeof(int32_t), cudaMemcpyDeviceToHost));
}

// A launch with programmatic stream serialization (see ref_wait_previous).
template <typename... KArgs, typename... Args>
static void ref_launch(void (*kernel)(KArgs...), int grid, int block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CS_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
}

// Frames k0 .. k0 + n - 1 of the call (itimes[k]) in one launch of the one-block form.
template <int KT>
static void ref_enqueue_block_k(DeviceRef* d, uint32_t k0, uint32_t n) {
    const RefParams& p = d->p;
    const RefSparse sp = ref_sparse(d);
    uint32_t rows = 0, stage_P = 0, other = 0;
    const size_t smem = ref_block_smem(d, sp, stage_P, rows, other);
    ref_sp_frames_block<KT><<<1, REF_BLOCK_THREADS, smem, d->stream>>>(
        p, sp, d->slots.p, d->occ.p, d->conc.p, (const uint32_t*)d->itimes.p, k0, n, d->dense_next ? 1u : 0u,
        d->dense_always ? 1u : 0u, d->stat.p, d->diag.p, d->flag.p, stage_P, rows, other);
    CS_LAUNCH_CHECK();
}

static void ref_enqueue_block(DeviceRef* d, uint32_t k0, uint32_t n) {
    if (n == 0) return;
    if (d->p.K == 16u) ref_enqueue_block_k<16>(d, k0, n);
    else if (d->p.K == 8u) ref_enqueue_block_k<8>(d, k0, n);
    else ref_enqueue_block_k<0>(d, k0, n);
    d->dense_next = false;
    d->rows_stale = true;
}

template <int KT>
static void ref_enqueue_frame_k(DeviceRef* d, uint32_t k) {
    const RefParams& p = d->p;
    const RefSparse sp = ref_sparse(d);
    uint32_t rows = 0, stage_P = 0;
    const size_t range = ref_range_words(sp.cw) * 4, P = ref_P_smem(p, stage_P);
    const size_t smem = ref_cme_smem(p, sp, REF_NT, 0, REF_SMEM, rows);
    const int grid = (int)std::min<uint32_t>((sp.W + sp.cw - 1u) / sp.cw, 16u * (uint32_t)d->sms);
    const uint32_t dense = (d->dense_next || d->dense_always) ? 1u : 0u;
    ref_launch(ref_sp_directions<KT>, grid, REF_NT, range + P, d->stream, p, sp, (const uint8_t*)d->slots.p,
               (const uint32_t*)d->occ.p, (const uint32_t*)d->itimes.p, k, d->diag.p, d->flag.p, stage_P);
    ref_launch(ref_sp_move<KT>, grid, REF_NT, range, d->stream, p, sp, d->slots.p, d->occ.p, d->conc.p, d->diag.p,
               (const uint32_t*)d->flag.p);
    ref_launch(ref_sp_cme<KT>, grid, REF_NT, smem, d->stream, p, sp, d->slots.p, d->occ.p, d->conc.p,
               (const uint32_t*)d->itimes.p, k, dense, d->stat.p, d->diag.p, d->flag.p, rows);
}

static void ref_enqueue_frame(DeviceRef* d, uint32_t k) {
    if (d->p.K == 16u) ref_enqueue_frame_k<16>(d, k);
    else if (d->p.K == 8u) ref_enqueue_frame_k<8>(d, k);
    else ref_enqueue_frame_k<0>(d, k);
    d->dense_next = false;
    d->rows_stale = true;
}

static void ref_enqueue(DeviceRef* d, uint32_t n) {
    if (ref_one_block(d)) {
        ref_enqueue_block(d, 0, n);
        return;
    }
    for (uint32_t k = 0; k < n; k++) ref_enqueue_frame(d, k);
}

void ref_step(DeviceRef* d, uint32_t n_steps, const uint32_t* itimes, uint64_t frame0, uint32_t write_freq,
              const std::vector<uint32_t>& logging, std::vector<cs_stat_sample>& samples) {
    DeviceGuard g(d->device);
    if (n_steps == 0) return;
    const RefParams& p = d->p;
    // frames f in [frame0, frame0+n) sample before executing when f > 0 and f % write_freq == 0
    std::vector<uint64_t> sample_frames;
    if (write_freq)
        for (uint64_t f = frame0; f < frame0 + n_steps; f++)
            if (f > 0 && f % write_freq == 0) sample_frames.push_back(f);
    if (d->itimes.n < n_steps) d->itimes.alloc(std::max<uint32_t>(n_steps, 64));
    CS_CUDA(cudaMemcpyAsync(d->itimes.p, itimes, n_steps * sizeof(uint32_t), cudaMemcpyHostToDevice, d->stream));
    if (!sample_frames.empty() && d->sample_ring.n < sample_frames.size() * p.S1)
        d->sample_ring.alloc(sample_frames.size() * p.S1);
    size_t si = 0;
    uint32_t k0 = 0;  // first frame not yet enqueued (the one-block form runs the frames between samples)
    for (uint32_t k = 0; k < n_steps; k++) {
        uint64_t f = frame0 + k;
        if (si < sample_frames.size() && sample_frames[si] == f) {
            if (ref_one_block(d)) ref_enqueue_block(d, k0, k - k0);
            k0 = k;
            CS_CUDA(cudaMemcpyAsync(d->sample_ring.p + si * p.S1, d->stat.p, p.S1 * sizeof(int32_t),
                                    cudaMemcpyDeviceToDevice, d->stream));
            si++;
        }
        if (!ref_one_block(d)) ref_enqueue_frame(d, k);
    }
    if (ref_one_block(d)) ref_enqueue_block(d, k0, n_steps - k0);
    if (!sample_frames.empty()) {
        std::vector<int32_t> h(sample_frames.size() * p.S1);
        CS_CUDA(cudaMemcpyAsync(h.data(), d->sample_ring.p, h.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, d->stream));
        CS_CUDA(cudaStreamSynchronize(d->stream));
        for (size_t i = 0; i < sample_frames.size(); i++)
            for (uint32_t sp : logging)
                samples.push_back(cs_stat_sample{sp, h[i * p.S1 + sp], (uint32_t)sample_frames[i]});
    }
}

void ref_get_counts(DeviceRef* d, int64_t* counts) {
    DeviceGuard g(d->device);
    std::vector<int32_t> h(d->p.S1);
    CS_CUDA(cudaMemcpyAsync(h.data(), d->stat.p, h.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, d->stream));
    CS_CUDA(cudaStreamSynchronize(d->stream));
    for (uint32_t s = 0; s < d->p.S1; s++) counts[s] = h[s];
}

void ref_get_diag(DeviceRef* d, uint32_t* diag, uint32_t n) {
    DeviceGuard g(d->device);
    uint32_t h[DIAG_N];
    CS_CUDA(cudaMemcpyAsync(h, d->diag.p, sizeof(h), cudaMemcpyDeviceToHost, d->stream));
    CS_CUDA(cudaStreamSynchronize(d->stream));
    for (uint32_t i = 0; i < n; i++) diag[i] = i < DIAG_N ? h[i] : 0u;
}

void ref_sync(DeviceRef* d) {
    DeviceGuard g(d->device);
    CS_CUDA(cudaStreamSynchronize(d->stream));
}

}  // namespace cellsim

namespace cellsim {
float ref_time_frames(DeviceRef* d, uint32_t n, const uint32_t* itimes, uint64_t frame0) {
    DeviceGuard g(d->device);
    if (d->itimes.n < n) d->itimes.alloc(std::max<uint32_t>(n, 64));
    CS_CUDA(cudaMemcpyAsync(d->itimes.p, itimes, n * sizeof(uint32_t), cudaMemcpyHostToDevice, d->stream));
    CS_CUDA(cudaStreamSynchronize(d->stream));
    cudaEvent_t a, b;
    CS_CUDA(cudaEventCreate(&a));
    CS_CUDA(cudaEventCreate(&b));
    std::vector<cs_stat_sample> none;
    float ms = 0.0f;
    try {
        CS_CUDA(cudaEventRecord(a, d->stream));
        ref_enqueue(d, n);
        CS_CUDA(cudaEventRecord(b, d->stream));
        CS_CUDA(cudaEventSynchronize(b));
        CS_CUDA(cudaEventElapsedTime(&ms, a, b));
    } catch (...) {
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        throw;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    (void)frame0;
    return ms;
}
}  // namespace cellsim

// ------------------------------------------------------------------ allocation-free frame
//
// A reference-RNG frame on caller-owned device buffers that never allocates.
// It serves hosts that own all device memory themselves: an engine that
// reserves one arena at start-up and forbids further cudaMalloc (a cudaMalloc
// can synchronise the device and fragments that budget), or a real-time loop
// that cannot absorb an allocation's stall.  The only memory the frame needs
// beyond the caller's inputs and outputs (the per-slot direction bytes and the
// contention flag) lives in the fixed array below.  CUDA reserves that array
// on every GPU where this library's module is loaded, and it stays there until
// the process exits.
namespace cellsim {

constexpr size_t kNoAllocMaxSlots = (size_t)16 << 20;  // V * K <= 16 Mi slots (16 MiB of directions)
static __device__ __align__(256) uint8_t g_noalloc_scratch[kNoAllocMaxSlots + 256];

static std::mutex g_noalloc_mu;
static uint8_t* g_noalloc_addr[256];

// Device address of the scratch array on `device`, looked up once per device
// with that device current.
static uint8_t* noalloc_scratch(int device) {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (device < 0 || device >= 256) throw Error(CS_ERR_INVALID_ARG, "device ordinal out of range");
    if (!g_noalloc_addr[device]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) throw Error(CS_ERR_CUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
        g_noalloc_addr[device] = static_cast<uint8_t*>(p);
    }
    return g_noalloc_addr[device];
}

void ref_frame_noalloc(const cs_ref_frame_noalloc_args* a) {
    if (!a) throw Error(CS_ERR_INVALID_ARG, "args is NULL");
    const uint32_t K = a->max_particles_site;
    if (a->res[0] == 0 || a->res[1] == 0 || a->res[2] == 0) throw Error(CS_ERR_INVALID_ARG, "resolution must be positive");
    if (K < 1 || K > 16) throw Error(CS_ERR_LIMIT, "max_particles_site must be in 1..16");
    if (a->n_regions < 1 || a->n_regions > 256) throw Error(CS_ERR_LIMIT, "n_regions must be in 1..256");
    if (a->n_species > 255) throw Error(CS_ERR_LIMIT, "at most 255 species");
    if (a->n_reactions > 99) throw Error(CS_ERR_LIMIT, "at most 99 reactions");
    const uint64_t V = (uint64_t)a->res[0] * a->res[1] * a->res[2];
    if (V * K > kNoAllocMaxSlots)
        throw Error(CS_ERR_LIMIT, "cs_ref_frame_noalloc handles at most 16777216 slots (V*K); this lattice has " +
                                      std::to_string(V * K) + ": use cs_step, which allocates its own scratch");
    const void* ptrs[] = {a->slots_in, a->occupancy_in, a->conc_in, a->slots_out, a->occupancy_out, a->conc_out,
                          a->regions, a->reservoir, a->probabilities, a->stoich, a->reactants, a->rates, a->itime,
                          a->counts, a->diag};
    for (const void* q : ptrs)
        if (!q) throw Error(CS_ERR_INVALID_ARG, "every buffer pointer of cs_ref_frame_noalloc_args must be non-NULL");
    DeviceGuard g(a->device);
    uint8_t* scratch = noalloc_scratch(a->device);
    uint8_t* dirs = scratch;
    uint32_t* contended = reinterpret_cast<uint32_t*>(scratch + kNoAllocMaxSlots);
    RefParams p{};
    p.X = a->res[0]; p.Y = a->res[1]; p.Z = a->res[2];
    p.K = K; p.S1 = a->n_species + 1; p.R = a->n_reactions; p.NR = a->n_regions;
    p.YZ = p.Y * p.Z;
    p.V = V;
    p.tau = a->tau;
    p.P = a->probabilities;
    p.stoich = a->stoich;
    p.reactants = a->reactants;
    p.rates = a->rates;
    p.regions = a->regions;
    p.reservoir = a->reservoir;
    cudaStream_t st = static_cast<cudaStream_t>(a->stream);
    const int TB = 256;
    unsigned nb = (unsigned)((V + TB - 1) / TB);
    size_t smem = (p.S1 + 2) * sizeof(int32_t);
    // ref_directions rewrites every direction byte and clears the contention
    // flag before anything reads them, so stale scratch from an earlier call
    // never leaks into this frame.
    ref_directions<<<nb, TB, 0, st>>>(p, a->slots_in, a->occupancy_in, a->itime, 0u, dirs, a->diag, contended);
    ref_gather<<<nb, TB, 0, st>>>(p, a->slots_in, a->occupancy_in, a->conc_in, dirs, a->slots_out, a->occupancy_out,
                                  a->conc_out, contended);
    ref_serial_copy<<<std::min<unsigned>(nb, 4096u), TB, 0, st>>>(p, contended, a->slots_in, a->occupancy_in, a->conc_in,
                                                                  a->slots_out, a->occupancy_out, a->conc_out);
    ref_serial<<<1, 32, 0, st>>>(p, contended, a->slots_in, a->occupancy_in, dirs, a->slots_out, a->occupancy_out,
                                 a->conc_out, a->diag);
    ref_cme<<<nb, TB, smem, st>>>(p, a->slots_out, a->occupancy_out, a->conc_out, a->itime, 0u, a->counts, a->diag);
    CS_LAUNCH_CHECK();
}

}  // namespace cellsim
