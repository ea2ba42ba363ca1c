// device_inplace.cu — the kernels of the in-place sweep stream (see
// inplace_kernel.cuh for the scheme).
#include <cuda_runtime.h>

#include "cuda_check.h"
#include "inplace_kernel.cuh"
#include "prod_kernel.cuh"
#include "views.cuh"

namespace cellsim {

namespace {

constexpr int LINE_NT = 256, ROW_NT = INPLACE_THREADS;  // threads of a block of the X and Y sweeps / of the row kernel
constexpr int CAP = 1024;  // entries of a block's item list: (word << 5) | bit
constexpr int SNAP_BYTES = 4096;  // snapshots kept in shared memory (SNAP_BYTES / (K + 4) voxels)

// Areas of a unit's words in shared memory: occupied voxels and voxels of two or more particles (as the
// sweep started, then as the general path leaves them), voxels that may react, movers down and up, the
// voxels whose content the general path replaced, the rank of the word's first voxel on that path and
// those voxels, and the bits of the decisions made by the block; row units also keep where each word
// lies.  A row unit's sweep is over when its next-frame decisions are made, so those share its areas.
enum : int { W_OCC, W_MUL, W_RE, W_M, W_P, W_CLR, W_BASE, W_REST, W_Z0, W_Z1, W_Y0, W_Y1 };
enum : int { R_Z0 = W_M, R_Z1 = W_P, R_Y0 = W_CLR, R_Y1 = W_BASE, R_X0 = W_REST, R_X1 = W_REST + 1, R_INFO };
constexpr int areas_of(int axis) { return axis == 0 ? W_Y1 + 1 : axis == 1 ? W_Z1 + 1 : R_INFO + 1; }
// decision areas {down, up} of axis a in a line unit and in the decisions of a row unit
template <bool ROW>
__device__ __forceinline__ constexpr int area_of(int a) {
    return ROW ? (a == 0 ? R_X0 : a == 1 ? R_Y0 : R_Z0) : (a == 1 ? W_Y0 : W_Z0);
}
constexpr int N_QUIET = 17;  // quiet thresholds by particle number

// words of one block's shared memory; stride: words per area
__host__ __device__ constexpr size_t smem_words(int axis, int stride) {
    return (size_t)areas_of(axis) * stride + CAP / 2 + SNAP_BYTES / 4 + 16 + PD_N + N_QUIET + 3;
}

__device__ __forceinline__ void ip_allow_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void ip_wait_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Starts a load whose line is read later (the value is dropped).
template <typename V>
__device__ __forceinline__ void ip_touch(const V* p) {
    uint32_t d;
    asm volatile("ld.global.u32 %0, [%1];\n" : "=r"(d) : "l"(p));
}

// Voxel contents written in this launch by other threads of the block are read too, so these are
// ordinary loads (not the read-only path).
template <int K>
__device__ __forceinline__ Vox<K> ip_load(const uint8_t* lat, uint64_t v) {
    Vox<K> c;
    if constexpr (K == 16) {
        const uint4 t = *reinterpret_cast<const uint4*>(lat + v * 16);
        c.w[0] = (uint64_t)t.x | ((uint64_t)t.y << 32);
        c.w[1] = (uint64_t)t.z | ((uint64_t)t.w << 32);
    } else {
        const uint2 t = *reinterpret_cast<const uint2*>(lat + v * 8);
        c.w[0] = (uint64_t)t.x | ((uint64_t)t.y << 32);
    }
    return c;
}

template <int K>
__device__ __forceinline__ bool ip_equal(const Vox<K>& a, const Vox<K>& b) {
    uint64_t d = 0;
#pragma unroll
    for (int i = 0; i < K / 8; i++) d |= a.w[i] ^ b.w[i];
    return d == 0;
}

// What a block knows of its replicate.
struct Where {
    const uint32_t* thr;
    const uint32_t* quiet;    // [S1] quiet thresholds of one particle (shared memory)
    const uint32_t* quiet_n;  // [N_QUIET] quiet thresholds of any n particles (shared memory)
    const uint8_t* rpad;      // region codes of the replicate
    uint32_t X, Y, Z, Zr, S1, NC;
    uint32_t k0, k1;
};

// Where a word lies: its region code if its window has one (else 0), the sides on which its voxels
// have neighbours along x and y, whether its first voxel is the row's first, and the bit of the row's
// last voxel (63: in a later word).
constexpr uint32_t UNIFORM = 0x2000u;  // in a voxel's copy of the info, see decide_single
constexpr uint32_t IN_XL = 0x100u, IN_XH = 0x200u, IN_YL = 0x400u, IN_YH = 0x800u, IN_ZL = 0x1000u;
constexpr uint32_t INSIDE = IN_XL | IN_XH | IN_YL | IN_YH | IN_ZL | 63u << 16;  // neighbours on every side
__device__ __forceinline__ uint32_t word_info(const Where& W, uint32_t uc, uint32_t x, uint32_t y, uint32_t kk) {
    const uint32_t last = W.Z - 1u - 32u * kk;
    return uc | (x > 0u ? IN_XL : 0u) | (x + 1u < W.X ? IN_XH : 0u) | (y > 0u ? IN_YL : 0u) |
           (y + 1u < W.Y ? IN_YH : 0u) | (kk > 0u ? IN_ZL : 0u) | (min(last, 63u) << 16);
}

// Threshold rows (offsets into the table) of the moves along axes A0 .. 2 from a voxel (bit b of a word
// with info `info`, its region code at rpad[rp]).  Row 0 (region code 0, outside the lattice) is all zero.
struct Rows {
    uint32_t lo[3], hi[3];
};
template <int A0>
__device__ __forceinline__ Rows rows_of(const Where& W, uint32_t info, uint32_t rp, uint32_t b) {
    Rows r;
    const uint32_t uc = info & 0xFFu;
    const bool in[6] = {(info & IN_XL) != 0u, (info & IN_XH) != 0u, (info & IN_YL) != 0u, (info & IN_YH) != 0u,
                        b > 0u || (info & IN_ZL), b != info >> 16};
    if (uc) {
        const uint32_t row = (uc * W.NC + uc) * W.S1;
#pragma unroll
        for (int a = A0; a < 3; a++) {
            r.lo[a] = in[2 * a] ? row : 0u;
            r.hi[a] = in[2 * a + 1] ? row : 0u;
        }
    } else {
        const uint8_t* p = W.rpad + rp;
        const uint32_t row0 = (uint32_t)__ldg(p) * W.NC;
        const int64_t st[3] = {(int64_t)W.Y * W.Zr, (int64_t)W.Zr, 1};
#pragma unroll
        for (int a = A0; a < 3; a++) {
            r.lo[a] = in[2 * a] ? (row0 + (uint32_t)__ldg(p - st[a])) * W.S1 : 0u;
            r.hi[a] = in[2 * a + 1] ? (row0 + (uint32_t)__ldg(p + st[a])) * W.S1 : 0u;
        }
    }
    return r;
}

// Move masks of axes A0 .. 2 for a voxel of content c (n particles, n > 0): bit s of d[a] = slot s
// moves down along a, bit 16 + s = up, as decide_moves; b0 is B(v, 0).
template <int K, int A0>
__device__ __forceinline__ void decide_axes(const Where& W, const Rows& R, const Vox<K>& c, uint32_t n, uint32_t v,
                                            uint32_t frame, const U4& b0, uint32_t (&d)[3]) {
#pragma unroll
    for (int a = A0; a < 3; a++) d[a] = 0u;
    for (uint32_t s = 0; s < n; s++) {
        const uint32_t q = vox_get<K>(c, s);
        uint32_t tm[3], tp[3], any = 0u;
#pragma unroll
        for (int a = A0; a < 3; a++) {
            tm[a] = W.thr[R.lo[a] + q];
            tp[a] = W.thr[R.hi[a] + q];
            any |= tm[a] | tp[a];
        }
        if (any == 0u) continue;
        const U4 u = s == 0u ? b0 : d_philox(v, frame, s, 0u, W.k0, W.k1);
#pragma unroll
        for (int a = A0; a < 3; a++) {
            const uint32_t w = a == 0 ? u.x : a == 1 ? u.y : u.z;
            if (w < tm[a]) d[a] |= 1u << s;
            else if (w - tm[a] < tp[a]) d[a] |= 1u << (16 + s);
        }
    }
}

// Decisions of axes A0 .. 2 and the quiet test of a voxel whose only particle is q, into the decision
// areas of word idx.
template <int A0, bool ROW, int T>
__device__ __forceinline__ void decide_single(const Where& W, uint32_t q, uint32_t v, uint32_t info, uint32_t rp, uint32_t b,
                                              uint32_t frame, bool no_calm, uint32_t* acc, uint32_t idx) {
    const U4 b0 = d_philox(v, frame, 0u, 0u, W.k0, W.k1);
    const uint32_t bit = 1u << b;
    uint32_t uc = info & 0xFFu;
    if (info & UNIFORM) {  // the voxel and its six neighbours have one code, whatever its word's window has
        uc = __ldg(W.rpad + rp);
        info = INSIDE;
        b = 1u;
    }
    uint32_t tm[3], tp[3];
    if (uc) {  // one region around: one threshold, or 0 towards the lattice's faces
        const uint32_t t = W.thr[(uc * W.NC + uc) * W.S1 + q];
        tm[0] = info & IN_XL ? t : 0u;
        tp[0] = info & IN_XH ? t : 0u;
        tm[1] = info & IN_YL ? t : 0u;
        tp[1] = info & IN_YH ? t : 0u;
        tm[2] = b > 0u || (info & IN_ZL) ? t : 0u;
        tp[2] = b != info >> 16 ? t : 0u;
    } else {
        const Rows R = rows_of<A0>(W, info, rp, b);
#pragma unroll
        for (int a = A0; a < 3; a++) {
            tm[a] = W.thr[R.lo[a] + q];
            tp[a] = W.thr[R.hi[a] + q];
        }
    }
#pragma unroll
    for (int a = A0; a < 3; a++) {
        const uint32_t w = a == 0 ? b0.x : a == 1 ? b0.y : b0.z;
        const bool down = w < tm[a];
        // tm <= w < tm + tp moves up (tm + tp may be 2^32)
        if (down || w - tm[a] < tp[a]) atomicOr(acc + (area_of<ROW>(a) + (down ? 0 : 1)) * T + idx, bit);
    }
    if (!no_calm && (b0.w >> 8) + 1u > W.quiet[q]) atomicOr(acc + W_RE * T + idx, bit);
}

// calm_voxel, for three or more particles after the threshold of their number (the largest propensity
// any n particles can have)
template <int K>
__device__ __forceinline__ bool ip_calm(const ProdTables& T, const Where& W, uint32_t ci, const Vox<K>& c, uint32_t w3) {
    const uint32_t n = vox_n<K>(c);
    if (n >= 3u && (w3 >> 8) + 1u <= W.quiet_n[n]) return true;
    return calm_voxel<K>(c, w3, T.quiet + (size_t)ci * T.S1 * T.QS, T.QS, T.one + (size_t)ci * T.S1 * 3, T.g23 + 2 * ci,
                         T.a2 ? T.a2 + (size_t)ci * T.S1 * T.S1 : nullptr, T.tau);
}

// The same for a voxel of any content c (not empty): also its move masks in dec.
template <int K, int A0, bool ROW, int T>
__device__ __forceinline__ void decide_content(const InplaceParams& P, const Where& W, uint32_t ci, const Vox<K>& c,
                                               uint32_t v, uint64_t g, uint32_t info, uint32_t rp, uint32_t b,
                                               uint32_t frame, bool no_calm, uint32_t* acc, uint32_t idx) {
    const U4 b0 = d_philox(v, frame, 0u, 0u, W.k0, W.k1);
    const uint32_t n = vox_n<K>(c), bit = 1u << b;
    if (!no_calm && !ip_calm<K>(P.T, W, ci, c, b0.w)) atomicOr(acc + W_RE * T + idx, bit);
    if constexpr (A0 < 3) {
        const Rows R = rows_of<A0>(W, info, rp, b);
        uint32_t d[3];
        decide_axes<K, A0>(W, R, c, n, v, frame, b0, d);
#pragma unroll
        for (int a = A0; a < 3; a++) {
            if (d[a] == 0u) continue;
            if (d[a] & 0xFFFFu) atomicOr(acc + area_of<ROW>(a) * T + idx, bit);
            if (d[a] >> 16) atomicOr(acc + (area_of<ROW>(a) + 1) * T + idx, bit);
            if (n > 1u) P.dec[a][g] = d[a];
        }
    }
}

// The content of a voxel: species byte sp where it holds one particle, its slots where it holds more.
template <int K>
__device__ __forceinline__ Vox<K> content_of(const uint8_t* lat, const uint8_t* sp, uint32_t v, bool occupied, bool multi) {
    if (multi) return ip_load<K>(lat, v);
    Vox<K> c = vox_zero<K>();
    if (occupied) c.w[0] = *sp;
    return c;
}
template <int K>
__device__ __forceinline__ void store_content(uint8_t* lat, uint8_t* sp, uint32_t v, const Vox<K>& c) {
    if (vox_n<K>(c) > 1u) st_vox_g<K>(lat + (uint64_t)v * K, c);
    else *sp = (uint8_t)c.w[0];
}

// Ranks of the thread's items among the block's (thread order) for counts packed in one word, and
// their totals; every thread calls it.  tmp: a shared word per warp, free again after the caller's next
// barrier.
template <int NT, typename C>
__device__ __forceinline__ C block_rank(C cnt, C* tmp, C& total) {
    constexpr int NWARP = NT / 32;
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    C incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const C u = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += u;
    }
    if (lane == 31u) tmp[w] = incl;
    __syncthreads();
    C off = 0;
    total = 0;
#pragma unroll
    for (int i = 0; i < NWARP; i++) {
        const C t = tmp[i];
        if (i < (int)w) off += t;
        total += t;
    }
    return off + incl - cnt;
}

// Lists the thread's items (bits of mask[s], word s * NT + tid) whose rank lies in [from, from + CAP).
template <int NT, int NW>
__device__ __forceinline__ void put_items(const uint32_t (&mask)[NW], uint32_t rank, uint32_t from, uint16_t* list) {
#pragma unroll
    for (int s = 0; s < NW; s++) {
        const uint32_t idx = (uint32_t)s * NT + threadIdx.x;
        for (uint32_t m = mask[s]; m; m &= m - 1u) {
            const uint32_t k = rank++ - from;
            if (k < (uint32_t)CAP) list[k] = (uint16_t)((idx << 5) | (uint32_t)(__ffs((int)m) - 1));
        }
    }
}

// The words of one voxel word and its neighbours along the axis as the sweep started: own (o, u, m,
// p), at -1 and +1 (o, u, m, p), at -2 (p) and +2 (m), each aligned to the own bits.
struct Around {
    uint32_t o, u, m, p, ol, ul, pl, oh, uh, mh, pll, mhh;
};
// Simple moves out of the word (down, up), the empty voxels of the word that simple moves fill, and
// the other voxels that lose or receive a particle.
struct Moves {
    uint32_t down, up, fill, rest;
};
__device__ __forceinline__ Moves moves_of(const Around& A) {
    Moves r;
    const uint32_t single = A.o & ~A.u, arrive = A.pl | A.mh;
    r.down = A.m & single & ~arrive & ~A.ol & ~A.pll;
    r.up = A.p & single & ~arrive & ~A.oh & ~A.mhh;
    // a mover of the lower (upper) neighbour for which this voxel is the empty, sole target
    const uint32_t from_l = A.pl & A.ol & ~A.ul & ~(A.pll | A.m) & ~A.o & ~A.mh;
    const uint32_t from_h = A.mh & A.oh & ~A.uh & ~(A.mhh | A.p) & ~A.o & ~A.pl;
    r.fill = from_l | from_h;
    r.rest = (A.m | A.p | arrive) & ~(r.down | r.up | r.fill);
    return r;
}

// A listed voxel: replicate-relative voxel and word, its word's info and the mover bits around it.
struct Site {
    uint32_t v, word, info, rp;
    bool m, p, from_lo, from_hi;  // own movers down / up; a mover of the lower / upper neighbour comes here
};

// One sweep of a unit along axis AX, in place.  simple / rest: the simple moves out of the thread's
// words (s * NT + tid; the areas W_M and W_P tell their direction) and the other voxels that lose or
// receive particles.  at(idx, b) describes a voxel; target(idx, b, down) steps (idx, b) to the
// neighbour.  Later decisions (axes AX + 1 .. 2, and the quiet test unless no_calm) go to the decision
// areas; for the general path the content areas are filled too.
template <int K, int AX, int NT, int NW, typename At, typename Target>
__device__ __forceinline__ void sweep_unit(const InplaceParams& P, const Where& W, const RepDesc& rd,
                                           const uint32_t (&simple)[NW], const uint32_t (&rest)[NW], uint32_t rank,
                                           uint32_t total, uint32_t* acc, uint16_t* list, uint8_t* s_snap,
                                           uint32_t frame, uint32_t stride, At at, Target target) {
    constexpr int T = NW * NT;
    const bool no_calm = P.T.n_zero_order != 0u;
    const uint32_t ns = total & 0xFFFFu, nr = total >> 16;
    const uint32_t rank_s = rank & 0xFFFFu, rank_r = rank >> 16;
    const bool one_list = ns + nr <= (uint32_t)CAP;
    // few enough voxels on the general path: their snapshots and move masks in shared memory
    constexpr uint32_t SNAPS = SNAP_BYTES / (K + 4);
    const bool local = nr <= SNAPS;
    uint32_t* const s_dec = reinterpret_cast<uint32_t*>(s_snap + SNAPS * K);
    if (nr) {
        uint32_t r = rank_r;
#pragma unroll
        for (int s = 0; s < NW; s++) {
            const uint32_t idx = (uint32_t)s * NT + threadIdx.x;
            acc[W_REST * T + idx] = rest[s];
            acc[W_BASE * T + idx] = r;
            r += (uint32_t)__popc(rest[s]);
        }
    }
    uint8_t* const lat = P.lat + rd.base * K;
    uint8_t* const snap = P.snap + rd.base * K;
    uint8_t* const spec = P.spec + rd.obase * 32u;
    // phase 0: the simple moves, and snapshots of the other voxels; phase 1: their new contents
    for (uint32_t phase = 0; phase < 2u; phase++) {
        const uint32_t first = phase && one_list ? ns : 0u;  // list entry of the first item
        const uint32_t n_all = phase ? nr : ns + nr;
        for (uint32_t from = 0; from < n_all; from += CAP) {
            if (phase == 0u || !one_list) {
                if (from || phase) __syncthreads();
                if (phase == 0u) {
                    put_items<NT, NW>(simple, rank_s, from, list);
                    put_items<NT, NW>(rest, ns + rank_r, from, list);
                } else {
                    put_items<NT, NW>(rest, rank_r, from, list);
                }
                __syncthreads();
            }
            const uint32_t n = min(n_all - from, (uint32_t)CAP);
            for (uint32_t i = threadIdx.x; i < n; i += NT) {
                const uint32_t e = list[first + i];
                uint32_t idx = e >> 5, b = e & 31u;
                Site s = at(idx, b);
                if (phase == 0u && from + i < ns) {
                    const uint32_t q = spec[s.word * 32u + b];
                    target(idx, b, s.m);
                    s = at(idx, b);
                    spec[s.word * 32u + b] = (uint8_t)q;
                    if constexpr (AX < 2) {
                        decide_single<AX + 1, false, T>(W, q, s.v, s.info, s.rp, b, frame, no_calm, acc, idx);
                    } else if (!no_calm) {
                        const U4 b0 = d_philox(s.v, frame, 0u, 0u, W.k0, W.k1);
                        if ((b0.w >> 8) + 1u > W.quiet[q]) atomicOr(acc + W_RE * T + idx, 1u << b);
                    }
                    continue;
                }
                const uint32_t v = s.v, bit = 1u << b;
                const uint64_t g = rd.base + v;
                const uint32_t* const dec = P.dec[AX];
                uint8_t* const sp = spec + (s.word * 32u + b);
                if (phase == 0u) {
                    const bool multi = acc[W_MUL * T + idx] & bit;
                    const uint32_t d = (s.m || s.p) ? (multi ? dec[g] : s.m ? 1u : 0x10000u) : 0u;
                    const Vox<K> c = content_of<K>(lat, sp, v, acc[W_OCC * T + idx] & bit, multi);
                    const uint32_t k = from + i - ns;
                    if (local) {
                        reinterpret_cast<Vox<K>*>(s_snap)[k] = c;
                        s_dec[k] = d;
                    } else {
                        st_vox_g<K>(snap + (uint64_t)v * K, c);
                    }
                    continue;
                }
                Vox<K> own, lo = vox_zero<K>(), hi = vox_zero<K>();
                uint32_t dme = 0u, dlo = 0u, dhi = 0u;
                if (local) {
                    auto rank_of = [&](uint32_t j, uint32_t c) -> uint32_t {
                        return acc[W_BASE * T + j] + (uint32_t)__popc(acc[W_REST * T + j] & ((1u << c) - 1u));
                    };
                    const Vox<K>* const sc = reinterpret_cast<const Vox<K>*>(s_snap);
                    own = sc[from + i];
                    dme = s_dec[from + i];
                    if (s.m || s.from_lo) {
                        uint32_t j = idx, c = b;
                        target(j, c, true);
                        const uint32_t k = rank_of(j, c);
                        lo = sc[k];
                        dlo = s.from_lo ? s_dec[k] : 0u;
                    }
                    if (s.p || s.from_hi) {
                        uint32_t j = idx, c = b;
                        target(j, c, false);
                        const uint32_t k = rank_of(j, c);
                        hi = sc[k];
                        dhi = s.from_hi ? s_dec[k] : 0u;
                    }
                } else {
                    own = ip_load<K>(snap, v);
                    if (s.m || s.from_lo) lo = ip_load<K>(snap, v - stride);
                    if (s.p || s.from_hi) hi = ip_load<K>(snap, v + stride);
                    if (s.m || s.p) dme = vox_n<K>(own) == 1u ? (s.m ? 1u : 0x10000u) : dec[g];
                    if (s.from_lo) dlo = vox_n<K>(lo) == 1u ? 0x10000u : dec[g - stride];
                    if (s.from_hi) dhi = vox_n<K>(hi) == 1u ? 1u : dec[g + stride];
                }
                const Vox<K> r = combine<K>(own, dme, lo, dlo, hi, dhi, v, v - stride, v + stride, frame, (uint32_t)AX);
                if (ip_equal<K>(r, own)) continue;  // every move refused for lack of room: the decisions stand
                const uint32_t n0 = vox_n<K>(own), n1 = vox_n<K>(r);
                atomicOr(acc + W_CLR * T + idx, bit);
                if ((n0 > 0u) != (n1 > 0u)) atomicXor(acc + W_OCC * T + idx, bit);
                if ((n0 > 1u) != (n1 > 1u)) atomicXor(acc + W_MUL * T + idx, bit);
                if (n1 == 0u) continue;
                store_content<K>(lat, sp, v, r);
                decide_content<K, AX + 1, false, T>(P, W, rd.counts_index, r, v, g, s.info, s.rp, b, frame, no_calm, acc, idx);
            }
        }
        if (phase == 0u && nr == 0u) break;
        __syncthreads();
    }
    __syncthreads();
}

// Starts the copies of replicate ri's tables to shared memory (complete after cp_async_wait<0> and a
// barrier).  No launch writes them, so they are read before the wait for the previous launch, and
// every copy is in flight at once: the block's first loads cost one L2 round trip, not one per table.
__device__ __forceinline__ void copy4(uint32_t* s, const uint32_t* g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_u32(s)), "l"(g) : "memory");
}
template <int NT>
__device__ __forceinline__ void stage_tables(const InplaceParams& P, uint32_t ri, uint32_t* s_tab, Where& W) {
    W.S1 = P.T.S1;
    W.NC = P.T.NC;
    uint32_t* const s_thr = s_tab;  // 16-byte aligned, as the table is
    W.thr = P.T.thr;
    uint32_t n = 0u;
    if (P.thr_smem) {
        n = W.NC * W.NC * W.S1;
        for (uint32_t i = threadIdx.x; i < n / 4u; i += NT) cp_async<16>(s_thr + 4u * i, P.T.thr + 4u * i, true);
        if (threadIdx.x < (n & 3u)) copy4(s_thr + (n & ~3u) + threadIdx.x, P.T.thr + (n & ~3u) + threadIdx.x);
        W.thr = s_thr;
    }
    W.quiet_n = s_tab + n;
    W.quiet = s_tab + n + N_QUIET;
    const uint32_t* const quiet = P.T.quiet + (size_t)ri * W.S1 * P.T.QS;
    if (threadIdx.x < N_QUIET) copy4(s_tab + n + threadIdx.x, P.T.quiet_n + (size_t)ri * N_QUIET + threadIdx.x);
    for (uint32_t i = threadIdx.x; i < W.S1; i += NT) copy4(s_tab + n + N_QUIET + i, quiet + i * P.T.QS);
    cp_async_commit();
}
__device__ __forceinline__ void set_where(const InplaceParams& P, const RepDesc& rd, Where& W) {
    W.rpad = P.region_pad + rd.rbase;
    W.X = rd.X;
    W.Y = rd.Y;
    W.Z = rd.Z;
    W.Zr = rd.Zr;
    W.k0 = rd.seed_lo;
    W.k1 = rd.seed_hi;
}

// The X (AX = 0) or Y (AX = 1) sweep of one unit of at most NW * NT words per block.
template <int K, int AX, int NW>
__global__ void __launch_bounds__(LINE_NT, 4) inplace_line_kernel(const __grid_constant__ InplaceParams P) {
    constexpr int NT = LINE_NT;
    constexpr int STR = NW * NT;
    extern __shared__ __align__(16) uint32_t sm[];
    uint32_t* const acc = sm;  // areas of STR words
    uint32_t* const tail = sm + areas_of(AX) * STR;
    uint16_t* const list = reinterpret_cast<uint16_t*>(tail);
    uint8_t* const s_snap = reinterpret_cast<uint8_t*>(tail + CAP / 2);
    uint32_t* const tmp = tail + CAP / 2 + SNAP_BYTES / 4;
    const uint32_t tid = threadIdx.x;
    Where W;
    ip_allow_next();
    const LineUnit U = P.units[blockIdx.x];
    const uint32_t ri = P.n_rep == 1u ? 0u : U.rep;
    const RepDesc rd = P.reps[ri];
    stage_tables<NT>(P, ri, tmp + 16 + PD_N, W);
    set_where(P, rd, W);
    ip_wait_previous();
    uint32_t frame = P.frame;
    if (!P.explicit_frame) {
        frame = AX == 0 ? *P.fa : *P.fb - 1u;
        if (blockIdx.x == 0 && tid == 0) *(AX == 0 ? P.fb : P.fa) = frame + 1u;
    }
    if (P.from && (int32_t)(frame - P.from[ri]) < 0) {
        cp_async_wait<0>();
        return;
    }
    const uint32_t lw = U.lw, pitch = 1u << lw, len = AX == 0 ? rd.X : rd.Y, T = len << lw;
    const uint32_t plane = rd.Y * rd.Wz;  // words of a plane
    // word idx: line position idx >> lw, column idx & (pitch - 1)
    auto word_of = [&](uint32_t idx) -> uint32_t {
        const uint32_t l = idx >> lw, c = idx & (pitch - 1u);
        return AX == 0 ? l * plane + U.a + c : (U.a * rd.Y + l) * rd.Wz + U.b + c;
    };
    uint2* const mv = P.mv[AX] + rd.obase;
    uint32_t any = 0u;
    {
        uint2 t[NW];
        uint32_t o[NW], u[NW];
#pragma unroll
        for (int s = 0; s < NW; s++) {
            const uint32_t idx = (uint32_t)s * NT + tid;
            t[s] = make_uint2(0u, 0u);
            o[s] = u[s] = 0u;
            if (idx < T && (idx & (pitch - 1u)) < U.n) {
                const uint32_t wo = word_of(idx);
                t[s] = mv[wo];
                o[s] = P.occ[rd.obase + wo];
                u[s] = P.mul[rd.obase + wo];
            }
        }
#pragma unroll
        for (int s = 0; s < NW; s++) {
            const uint32_t idx = (uint32_t)s * NT + tid;
            if (idx < T) {
                acc[W_M * STR + idx] = t[s].x;
                acc[W_P * STR + idx] = t[s].y;
                acc[W_OCC * STR + idx] = o[s];
                acc[W_MUL * STR + idx] = u[s];
                any |= t[s].x | t[s].y;
            }
        }
    }
    cp_async_wait<0>();
    if (!__syncthreads_or((int)(any != 0u))) return;  // nothing moves along the axis in these lines
    uint32_t simple[NW], rest[NW], fill[NW], cnt = 0u;
#pragma unroll
    for (int s = 0; s < NW; s++) {
        const uint32_t idx = (uint32_t)s * NT + tid;
        simple[s] = rest[s] = fill[s] = 0u;
        if (idx < T) {
            auto w = [&](int area, int step) -> uint32_t {
                const int j = (int)idx + step * (int)pitch;
                return j >= 0 && j < (int)T ? acc[area * STR + j] : 0u;
            };
            const uint32_t m = acc[W_M * STR + idx], p = acc[W_P * STR + idx], pl = w(W_P, -1), mh = w(W_M, 1);
            if (m | p | pl | mh) {
                const Around A{acc[W_OCC * STR + idx], acc[W_MUL * STR + idx], m, p, w(W_OCC, -1), w(W_MUL, -1), pl,
                               w(W_OCC, 1), w(W_MUL, 1), mh, w(W_P, -2), w(W_M, 2)};
                const Moves M = moves_of(A);
                simple[s] = M.down | M.up;
                rest[s] = M.rest;
                fill[s] = M.fill;
                cnt += (uint32_t)__popc(simple[s]) + ((uint32_t)__popc(rest[s]) << 16);
                acc[W_RE * STR + idx] = acc[W_CLR * STR + idx] = 0u;
#pragma unroll
                for (int k = W_Z0; k < areas_of(AX); k++) acc[k * STR + idx] = 0u;
            }
        }
    }
    uint32_t total;
    const uint32_t rank = block_rank<NT, uint32_t>(cnt, tmp, total);
    auto at = [&](uint32_t idx, uint32_t b) -> Site {
        Site s;
        const uint32_t bit = 1u << b, l = idx >> lw, c = idx & (pitch - 1u);
        uint32_t x, y, kk;
        if (AX == 0) {
            const uint32_t j = U.a + c;
            x = l;
            y = j / rd.Wz;
            kk = j - y * rd.Wz;
        } else {
            x = U.a;
            y = l;
            kk = U.b + c;
        }
        const uint32_t xy = x * rd.Y + y;
        const uint32_t z = 32u * kk + b;
        s.v = xy * rd.Z + z;
        s.word = xy * rd.Wz + kk;
        const uint32_t uc = (rd.flags & 1u) ? 1u : P.wcode ? (uint32_t)__ldg(P.wcode + rd.obase + s.word) : 0u;
        s.info = word_info(W, uc, x, y, kk);
        s.rp = xy * rd.Zr + z + 2u;
        s.m = (acc[W_M * STR + idx] & bit) != 0u;
        s.p = (acc[W_P * STR + idx] & bit) != 0u;
        s.from_lo = idx >= pitch && (acc[W_P * STR + idx - pitch] & bit);
        s.from_hi = idx + pitch < T && (acc[W_M * STR + idx + pitch] & bit);
        return s;
    };
    auto target = [&](uint32_t& idx, uint32_t&, bool down) { idx = down ? idx - pitch : idx + pitch; };
    sweep_unit<K, AX, NT, NW>(P, W, rd, simple, rest, rank, total, acc, list, s_snap, frame, AX == 0 ? rd.Y * rd.Z : rd.Z, at, target);
    // the words: used decisions cleared, occupancy and later decisions of the changed voxels replaced
    // (all loads before the stores, so that they are in flight together)
    uint2 y[NW], z[NW];
    uint32_t re[NW];
#pragma unroll
    for (int s = 0; s < NW; s++) {
        y[s] = z[s] = make_uint2(0u, 0u);
        re[s] = 0u;
        if (simple[s] | rest[s] | fill[s]) {
            const uint64_t gw = rd.obase + word_of((uint32_t)s * NT + tid);
            re[s] = P.react[gw];
            z[s] = P.mv[2][gw];
            if (AX == 0) y[s] = P.mv[1][gw];
        }
    }
#pragma unroll
    for (int s = 0; s < NW; s++) {
        const uint32_t idx = (uint32_t)s * NT + tid;
        if ((simple[s] | rest[s] | fill[s]) == 0u) continue;
        const uint32_t wo = word_of(idx);
        const uint64_t gw = rd.obase + wo;
        const uint32_t clr = acc[W_CLR * STR + idx] | simple[s];
        auto merge = [&](uint32_t old, int area) { return (old & ~clr) | acc[area * STR + idx]; };
        if (acc[W_M * STR + idx] | acc[W_P * STR + idx]) mv[wo] = make_uint2(0u, 0u);
        if (AX == 0) P.mv[1][gw] = make_uint2(merge(y[s].x, W_Y0), merge(y[s].y, W_Y1));
        P.mv[2][gw] = make_uint2(merge(z[s].x, W_Z0), merge(z[s].y, W_Z1));
        P.react[gw] = merge(re[s], W_RE);
        P.occ[gw] = (acc[W_OCC * STR + idx] & ~simple[s]) | fill[s];
        P.mul[gw] = acc[W_MUL * STR + idx];
    }
}

// Brings the reaction tables into the SM's L1 while the block sweeps, for the SSA of a voxel that may
// react: its chain reads about 15 entries one after another, an L2 round trip each if they are cold.
__device__ __forceinline__ void touch_tables(const ProdTables& T) {
    for (uint32_t i = 0; i < T.S1 * 16u; i += 128u) ip_touch(reinterpret_cast<const uint8_t*>(T.rmask) + i);
    for (uint32_t i = 0; i + 3u < T.R * 3u; i += 128u) ip_touch(T.rx_reactants + i);
    for (uint32_t i = 0; i < T.R; i += 32u) ip_touch(T.rx_rate + i);
    for (uint32_t i = 0; i < T.R * 8u; i += 128u) {
        ip_touch(T.rx_ch_sp + i);
        ip_touch(T.rx_ch_d + i);
    }
}

// The Z sweep of one unit of rows per block, the SSA of its voxels that may react and, for the next
// frame, the decisions of its occupied voxels.
template <int K>
__global__ void __launch_bounds__(ROW_NT, 7) inplace_row_kernel(const __grid_constant__ InplaceParams P) {
    constexpr int NT = ROW_NT, NWARP = NT / 32;
    constexpr int NW = INPLACE_ROW_WORDS / NT, STR = NW * NT;
    extern __shared__ __align__(16) uint32_t sm[];
    uint32_t* const acc = sm;  // areas of STR words
    uint32_t* const tail = sm + areas_of(2) * STR;
    uint16_t* const list = reinterpret_cast<uint16_t*>(tail);
    uint8_t* const s_snap = reinterpret_cast<uint8_t*>(tail + CAP / 2);
    uint32_t* const tmp = tail + CAP / 2 + SNAP_BYTES / 4;
    uint32_t* const s_diag = tmp + 16;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    Where W;
    ip_allow_next();
    const LineUnit U = P.units[blockIdx.x];
    const uint32_t ri = P.n_rep == 1u ? 0u : U.rep;
    const RepDesc rd = P.reps[ri];
    stage_tables<NT>(P, ri, s_diag + PD_N, W);
    set_where(P, rd, W);
    if (tid < PD_N) s_diag[tid] = 0u;
    const uint32_t Wz = rd.Wz, T = (uint32_t)U.n * Wz;
    const uint32_t w0 = U.a * Wz;  // the unit's words are consecutive
    const uint64_t gw0 = rd.obase + w0;
    const bool zero_order = P.T.n_zero_order != 0u;
    const uint32_t magic = (65536u + Wz - 1u) / Wz;  // idx / Wz = idx * magic >> 16 for idx < 512, Wz <= 32
    auto voxel_of = [&](uint32_t idx, uint32_t b) -> uint32_t {
        const uint32_t r = idx * magic >> 16;
        return (U.a + r) * rd.Z + 32u * (idx - r * Wz) + b;
    };
    const uint32_t x0 = U.a / rd.Y, y0 = U.a - x0 * rd.Y;
#pragma unroll
    for (int s = 0; s < NW; s++) {
        const uint32_t idx = (uint32_t)s * NT + tid;
        if (idx < T) {
            const uint32_t r = idx * magic >> 16, kk = idx - r * Wz;
            uint32_t x = x0, y = y0 + r;
            if (y >= rd.Y) {
                const uint32_t d = y / rd.Y;
                x += d;
                y -= d * rd.Y;
            }
            const uint32_t uc = (rd.flags & 1u) ? 1u : P.wcode ? (uint32_t)__ldg(P.wcode + gw0 + idx) : 0u;
            acc[R_INFO * STR + idx] = word_info(W, uc, x, y, kk);
        }
    }
    ip_wait_previous();
    uint32_t frame = P.frame;  // of the sweep; the decisions are for `next`
    if (!P.explicit_frame) frame = P.decide_only ? *P.fa : *P.fa - 1u;
    const uint32_t next = P.decide_only ? frame : frame + 1u;
    bool decide_only = P.decide_only != 0u;
    if (P.from) {
        const uint32_t from = P.from[ri];
        if ((int32_t)(next - from) < 0) {
            cp_async_wait<0>();
            return;
        }
        decide_only |= (int32_t)(frame - from) < 0;
    }
    uint2* const mv = P.mv[2] + gw0;
    uint8_t* const lat = P.lat + rd.base * K;
    uint8_t* const spec = P.spec + gw0 * 32u;
    // occupancy, multi-particle and reacting voxels of the thread's words; had: bit s = mv[2] of word
    // s, bit 8 + s = react of word s is set
    uint32_t o[NW], u[NW], re[NW], had = 0u;
    {
        uint2 t[NW];
#pragma unroll
        for (int s = 0; s < NW; s++) {
            const uint32_t idx = (uint32_t)s * NT + tid;
            o[s] = u[s] = re[s] = 0u;
            t[s] = make_uint2(0u, 0u);
            if (idx < T) {
                if (!decide_only) {
                    t[s] = mv[idx];
                    re[s] = P.react[gw0 + idx];
                }
                o[s] = P.occ[gw0 + idx];
                u[s] = P.mul[gw0 + idx];
            }
        }
#pragma unroll
        for (int s = 0; s < NW; s++) {
            const uint32_t idx = (uint32_t)s * NT + tid;
            if (idx < T) {
                if (t[s].x | t[s].y) had |= 1u << s;
                if (re[s]) {
                    had |= 0x100u << s;
                    touch_tables(P.T);
                }
                acc[W_M * STR + idx] = t[s].x;
                acc[W_P * STR + idx] = t[s].y;
                acc[W_OCC * STR + idx] = o[s];
                acc[W_MUL * STR + idx] = u[s];
            }
        }
    }
    cp_async_wait<0>();
    if (__syncthreads_or((int)(had != 0u || zero_order || P.resv_bits != nullptr) && !decide_only)) {
        uint32_t simple[NW], rest[NW], fill[NW], cnt = 0u;
#pragma unroll
        for (int s = 0; s < NW; s++) {
            const uint32_t idx = (uint32_t)s * NT + tid;
            simple[s] = rest[s] = fill[s] = 0u;
            if (idx < T) {
                const uint32_t info = acc[R_INFO * STR + idx];
                const uint32_t m = acc[W_M * STR + idx], p = acc[W_P * STR + idx];
                // the row's previous and next words
                const bool hl = info & IN_ZL, hh = info >> 16 >= 32u;
                const uint32_t p0 = hl ? acc[W_P * STR + idx - 1u] : 0u, m1 = hh ? acc[W_M * STR + idx + 1u] : 0u;
                if (m | p | (p0 >> 31) | (m1 & 1u)) {
                    const uint32_t o0 = hl ? acc[W_OCC * STR + idx - 1u] : 0u, o1 = hh ? acc[W_OCC * STR + idx + 1u] : 0u;
                    const uint32_t u0 = hl ? acc[W_MUL * STR + idx - 1u] : 0u, u1 = hh ? acc[W_MUL * STR + idx + 1u] : 0u;
                    const Around A{o[s], u[s], m, p, (o[s] << 1) | (o0 >> 31), (u[s] << 1) | (u0 >> 31),
                                   (p << 1) | (p0 >> 31), (o[s] >> 1) | (o1 << 31), (u[s] >> 1) | (u1 << 31),
                                   (m >> 1) | (m1 << 31), (p << 2) | (p0 >> 30), (m >> 2) | (m1 << 30)};
                    const Moves M = moves_of(A);
                    simple[s] = M.down | M.up;
                    rest[s] = M.rest;
                    fill[s] = M.fill;
                    cnt += (uint32_t)__popc(simple[s]) + ((uint32_t)__popc(rest[s]) << 16);
                }
                acc[W_CLR * STR + idx] = acc[W_RE * STR + idx] = 0u;
            }
        }
        uint32_t total;
        uint32_t rank = block_rank<NT, uint32_t>(cnt, tmp, total);
        if (total) {
            auto at = [&](uint32_t idx, uint32_t b) -> Site {
                Site s;
                s.v = voxel_of(idx, b);
                s.rp = 0u;  // no decision after the Z sweep looks a region up
                s.info = acc[R_INFO * STR + idx];
                s.word = w0 + idx;
                const bool hl = s.info & IN_ZL, hh = s.info >> 16 >= 32u;
                const uint32_t m = acc[W_M * STR + idx], p = acc[W_P * STR + idx];
                s.m = (m >> b) & 1u;
                s.p = (p >> b) & 1u;
                s.from_lo = b > 0u ? (p >> (b - 1u)) & 1u : hl && (acc[W_P * STR + idx - 1u] >> 31);
                s.from_hi = b < 31u ? (m >> (b + 1u)) & 1u : hh && (acc[W_M * STR + idx + 1u] & 1u);
                return s;
            };
            auto target = [&](uint32_t& idx, uint32_t& b, bool down) {
                const uint32_t k = (idx << 5 | b) + (down ? 0xFFFFFFFFu : 1u);
                idx = k >> 5;
                b = k & 31u;
            };
            sweep_unit<K, 2, NT, NW>(P, W, rd, simple, rest, rank, total, acc, list, s_snap, frame, 1u, at, target);
        }
        // the voxels that may react: an SSA each, by one warp
        cnt = 0u;
#pragma unroll
        for (int s = 0; s < NW; s++) {
            const uint32_t idx = (uint32_t)s * NT + tid;
            if (idx < T) {
                const uint32_t clr = acc[W_CLR * STR + idx] | simple[s];
                o[s] = (acc[W_OCC * STR + idx] & ~simple[s]) | fill[s];
                u[s] = acc[W_MUL * STR + idx];
                re[s] = (re[s] & ~clr) | acc[W_RE * STR + idx];
                if (P.resv_bits) re[s] |= P.resv_bits[gw0 + idx];
                if (zero_order) {
                    const uint32_t last = acc[R_INFO * STR + idx] >> 16;
                    re[s] = last >= 31u ? 0xFFFFFFFFu : (2u << last) - 1u;
                }
                cnt += (uint32_t)__popc(re[s]);
                acc[W_OCC * STR + idx] = o[s];
            }
        }
        __syncthreads();
        rank = block_rank<NT, uint32_t>(cnt, tmp, total);
        if (total) {
            for (uint32_t from = 0; from < total; from += CAP) {
                if (from) __syncthreads();
                put_items<NT, NW>(re, rank, from, list);
                __syncthreads();
                const uint32_t n = min(total - from, (uint32_t)CAP);
                for (uint32_t i = warp; i < n; i += NWARP) {
                    const uint32_t e = list[i], idx = e >> 5, b = e & 31u, bit = 1u << b;
                    const uint32_t v = voxel_of(idx, b);
                    // no other warp changes this voxel's bits
                    const bool occupied = acc[W_OCC * STR + idx] & bit, multi = acc[W_MUL * STR + idx] & bit;
                    uint8_t* const sp = spec + (idx * 32u + b);
                    Vox<K> r = content_of<K>(lat, sp, v, occupied, multi);
                    const uint32_t rv = P.reservoir ? (uint32_t)__ldg(P.reservoir + rd.base + v) : 0u;
                    const uint32_t w3 = d_philox(v, frame, 0u, 0u, W.k0, W.k1).w;
                    const bool fired =
                        react_voxel_warp<K>(r, rv, v, frame, W.k0, W.k1, rd.rate_mult, P.T, nullptr,
                                            P.counts + (size_t)rd.counts_index * W.S1, s_diag, w3);
                    __syncwarp();
                    if (lane == 0u && fired) {
                        store_content<K>(lat, sp, v, r);
                        if (vox_empty<K>(r)) atomicAnd(acc + W_OCC * STR + idx, ~bit);
                        else atomicOr(acc + W_OCC * STR + idx, bit);
                        if (vox_n<K>(r) > 1u) atomicOr(acc + W_MUL * STR + idx, bit);
                        else atomicAnd(acc + W_MUL * STR + idx, ~bit);
                    }
                    __syncwarp();
                }
            }
            __syncthreads();
#pragma unroll
            for (int s = 0; s < NW; s++) {
                const uint32_t idx = (uint32_t)s * NT + tid;
                if (idx < T) {
                    o[s] = acc[W_OCC * STR + idx];
                    u[s] = acc[W_MUL * STR + idx];
                }
            }
        }
#pragma unroll
        for (int s = 0; s < NW; s++)
            if (simple[s] | rest[s] | fill[s] | re[s]) {
                const uint64_t gw = gw0 + (uint32_t)s * NT + tid;
                P.occ[gw] = o[s];
                P.mul[gw] = u[s];
            }
        __syncthreads();  // the sweep's areas take the decisions from here on
    }
    // the next frame's decisions: first the voxels of one particle with one region around them, then the
    // others of one particle, then the voxels of more particles, so that warps mostly run one path
    unsigned long long cnt = 0ull;
    uint32_t one_c[NW], one_n[NW];
#pragma unroll
    for (int s = 0; s < NW; s++) {
        const uint32_t idx = (uint32_t)s * NT + tid, one = o[s] & ~u[s];
        one_c[s] = one_n[s] = 0u;
        if (idx < T) {
            // voxels with one region code around them, known from the word's or the voxel's own window
            const uint32_t known = acc[R_INFO * STR + idx] & 0xFFu ? 0xFFFFFFFFu : P.uni ? __ldg(P.uni + gw0 + idx) : 0u;
            one_c[s] = one & known;
            one_n[s] = one & ~known;
            cnt += (unsigned long long)__popc(one_c[s]) | ((unsigned long long)__popc(one_n[s]) << 20) |
                   ((unsigned long long)__popc(u[s]) << 40);
            acc[W_RE * STR + idx] = 0u;
#pragma unroll
            for (int k = R_Z0; k <= R_X1; k++) acc[k * STR + idx] = 0u;
        }
    }
    unsigned long long total;
    const unsigned long long rank = block_rank<NT, unsigned long long>(cnt, reinterpret_cast<unsigned long long*>(tmp), total);
    const uint32_t n_c = (uint32_t)total & 0xFFFFFu, n_1 = n_c + ((uint32_t)(total >> 20) & 0xFFFFFu);
    const uint32_t n_all = n_1 + (uint32_t)(total >> 40);
    for (uint32_t from = 0; from < n_all; from += CAP) {
        if (from) __syncthreads();
        put_items<NT, NW>(one_c, (uint32_t)rank & 0xFFFFFu, from, list);
        put_items<NT, NW>(one_n, n_c + ((uint32_t)(rank >> 20) & 0xFFFFFu), from, list);
        put_items<NT, NW>(u, n_1 + (uint32_t)(rank >> 40), from, list);
        __syncthreads();
        const uint32_t n = min(n_all - from, (uint32_t)CAP);
        for (uint32_t i = tid; i < n; i += NT) {
            const uint32_t e = list[i], idx = e >> 5, b = e & 31u;
            const uint32_t r = idx * magic >> 16, z = 32u * (idx - r * Wz) + b;
            const uint32_t v = (U.a + r) * rd.Z + z, rp = (U.a + r) * rd.Zr + z + 2u;
            uint32_t info = acc[R_INFO * STR + idx];
            if (from + i < n_c && (info & 0xFFu) == 0u) info = UNIFORM;
            if (from + i < n_1)
                decide_single<0, true, STR>(W, spec[e], v, info, rp, b, next, zero_order, acc, idx);
            else
                decide_content<K, 0, true, STR>(P, W, rd.counts_index, ip_load<K>(lat, v), v, rd.base + v, info, rp, b,
                                                next, zero_order, acc, idx);
        }
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < NW; s++) {
        const uint32_t idx = (uint32_t)s * NT + tid;
        if (idx >= T) continue;
        const uint2 x = make_uint2(acc[R_X0 * STR + idx], acc[R_X1 * STR + idx]);
        const uint2 y = make_uint2(acc[R_Y0 * STR + idx], acc[R_Y1 * STR + idx]);
        const uint2 z = make_uint2(acc[R_Z0 * STR + idx], acc[R_Z1 * STR + idx]);
        const uint32_t r = acc[W_RE * STR + idx];
        if (x.x | x.y) P.mv[0][gw0 + idx] = x;
        if (y.x | y.y) P.mv[1][gw0 + idx] = y;
        if ((z.x | z.y) || (had >> s & 1u)) mv[idx] = z;
        if (r || (had >> (8 + s) & 1u)) P.react[gw0 + idx] = r;
    }
    if (tid < PD_N && s_diag[tid]) atomicAdd(P.diag + tid, s_diag[tid]);
}

// View 0 (views.cuh) of one replicate: a warp takes 32 words, their bitmap words one per lane, then word by
// word; the slots are read only of voxels of more particles.
template <int K>
__global__ void __launch_bounds__(256) inplace_view_kernel(const InplaceParams P, RepDesc rd, float* out, uint32_t per) {
    const uint32_t lane = threadIdx.x & 31u, bit = 1u << lane, words = rd.X * rd.Y * rd.Wz;
    for (uint32_t w0 = (blockIdx.x * 8u + (threadIdx.x >> 5)) * per; w0 < words; w0 += gridDim.x * 8u * per) {
        const uint32_t w = w0 + lane, n = min(per, words - w0);
        const uint32_t o = lane < n ? P.occ[rd.obase + w] : 0u, u = lane < n ? P.mul[rd.obase + w] : 0u;
        uint32_t row = w0 / rd.Wz, kk = w0 - row * rd.Wz;
#pragma unroll 8
        for (uint32_t j = 0; j < n; j++) {
            const uint32_t oj = __shfl_sync(0xffffffffu, o, (int)j), uj = __shfl_sync(0xffffffffu, u, (int)j);
            const uint32_t z = 32u * kk + lane;
            if (z < rd.Z) {
                uint32_t q = oj & bit ? P.spec[(rd.obase + w0 + j) * 32u + lane] : 0u;
                const uint64_t v = (uint64_t)row * rd.Z + z;
                if (uj & bit) q = view_majority<K>(ip_load<K>(P.lat, rd.base + v).w);
                out[v] = __fdiv_rn((float)q, 255.0f);
            }
            if (++kk == rd.Wz) {
                kk = 0u;
                row++;
            }
        }
    }
}

// Region windows of a single lattice, one warp per word: wcode, the code that every lattice voxel of the
// word's window (rows x-1 .. x+1, y-1 .. y+1, z from 32k-1 to 32k+32) shares, or 0; uni, the voxels whose
// six neighbours lie in the lattice and have the voxel's own code.
__global__ void __launch_bounds__(256) region_window_kernel(const uint8_t* rpad, RepDesc rd, uint8_t* wcode, uint32_t* uni) {
    const uint32_t lane = threadIdx.x & 31u, words = rd.X * rd.Y * rd.Wz;
    for (uint32_t w = blockIdx.x * 8u + (threadIdx.x >> 5); w < words; w += gridDim.x * 8u) {
        const uint32_t row = w / rd.Wz, k = w - row * rd.Wz, x = row / rd.Y, y = row - x * rd.Y, z = 32u * k + lane;
        auto code = [&](int dx, int dy, int dz) -> uint32_t {  // 0 outside the lattice
            const int xx = (int)x + dx, yy = (int)y + dy, zz = (int)z + dz;
            if ((unsigned)xx >= rd.X || (unsigned)yy >= rd.Y || (unsigned)zz >= rd.Z) return 0u;
            return __ldg(rpad + ((uint64_t)xx * rd.Y + (uint64_t)yy) * rd.Zr + (uint32_t)zz + 2u);
        };
        const uint32_t own = code(0, 0, 0), c = __shfl_sync(0xffffffffu, own, 0);
        bool same = true;
        for (int dx = -1; dx <= 1; dx++)
            for (int dy = -1; dy <= 1; dy++) {
                const uint32_t a = code(dx, dy, 0);
                same &= a == 0u || a == c;
                if (lane == 0u || lane == 31u) {
                    const uint32_t e = code(dx, dy, lane ? 1 : -1);
                    same &= e == 0u || e == c;
                }
            }
        same = __all_sync(0xffffffffu, same);
        const bool u = own && code(-1, 0, 0) == own && code(1, 0, 0) == own && code(0, -1, 0) == own &&
                       code(0, 1, 0) == own && code(0, 0, -1) == own && code(0, 0, 1) == own;
        const uint32_t m = __ballot_sync(0xffffffffu, u);
        if (lane == 0u) {
            wcode[w] = same ? (uint8_t)c : (uint8_t)0u;
            uni[w] = m;
        }
    }
}

// The state of the form from the slots: occupancy, voxels of two or more particles and the species
// bytes; a warp per row, blockIdx.y over the replicates.
template <int K>
__global__ void __launch_bounds__(256) inplace_pack_kernel(const InplaceParams P) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t rep = blockIdx.y; rep < P.n_rep; rep += gridDim.y) {
        const RepDesc rd = P.reps[rep];
        const uint32_t rows = rd.X * rd.Y;
        for (uint32_t row = blockIdx.x * 8u + (threadIdx.x >> 5); row < rows; row += gridDim.x * 8u)
            for (uint32_t k = 0; k < rd.Wz; k++) {
                const uint32_t z = 32u * k + lane;
                const Vox<K> c = z < rd.Z ? ip_load<K>(P.lat, rd.base + (uint64_t)row * rd.Z + z) : vox_zero<K>();
                const uint32_t n = vox_n<K>(c);
                const uint32_t o = __ballot_sync(0xffffffffu, n > 0u), u = __ballot_sync(0xffffffffu, n > 1u);
                const uint64_t gw = rd.obase + (uint64_t)row * rd.Wz + k;
                if (o) P.spec[gw * 32u + lane] = (uint8_t)c.w[0];
                if (lane == 0u) {
                    P.occ[gw] = o;
                    P.mul[gw] = u;
                }
            }
    }
}

// The slots of every voxel that does not hold two or more particles (those hold theirs already).
template <int K>
__global__ void __launch_bounds__(256) inplace_unpack_kernel(const InplaceParams P) {
    const uint32_t lane = threadIdx.x & 31u, bit = 1u << lane;
    for (uint32_t rep = blockIdx.y; rep < P.n_rep; rep += gridDim.y) {
        const RepDesc rd = P.reps[rep];
        const uint32_t rows = rd.X * rd.Y;
        for (uint32_t row = blockIdx.x * 8u + (threadIdx.x >> 5); row < rows; row += gridDim.x * 8u)
            for (uint32_t k = 0; k < rd.Wz; k++) {
                const uint32_t z = 32u * k + lane;
                const uint64_t gw = rd.obase + (uint64_t)row * rd.Wz + k;
                const uint32_t o = P.occ[gw], u = P.mul[gw];
                if (z >= rd.Z || (u & bit)) continue;
                Vox<K> c = vox_zero<K>();
                if (o & bit) c.w[0] = P.spec[gw * 32u + lane];
                st_vox_g<K>(P.lat + (rd.base + (uint64_t)row * rd.Z + z) * K, c);
            }
    }
}

// nw: words per thread of a line unit (1, 2 or 4)
template <int K, int AX>
void* line_kernel(int nw) {
    return nw == 1   ? reinterpret_cast<void*>(&inplace_line_kernel<K, AX, 1>)
           : nw == 2 ? reinterpret_cast<void*>(&inplace_line_kernel<K, AX, 2>)
                     : reinterpret_cast<void*>(&inplace_line_kernel<K, AX, 4>);
}
void* kernel_of(int K, int axis, int nw) {
    if (axis == 2)
        return K == 16 ? reinterpret_cast<void*>(&inplace_row_kernel<16>) : reinterpret_cast<void*>(&inplace_row_kernel<8>);
    if (axis == 1) return K == 16 ? line_kernel<16, 1>(nw) : line_kernel<8, 1>(nw);
    return K == 16 ? line_kernel<16, 0>(nw) : line_kernel<8, 0>(nw);
}

}  // namespace

void inplace_set_attrs() {
    for (int K : {8, 16})
        for (int axis = 0; axis < 3; axis++)
            for (int nw : {1, 2, 4}) {
                void* fn = kernel_of(K, axis, nw);
                CS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
                CS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
            }
}

void inplace_launch(int K, int axis, uint32_t grid, uint32_t words, cudaStream_t s, const InplaceParams& P) {
    if (grid == 0) return;
    const int nt = axis == 2 ? ROW_NT : LINE_NT;
    const int nw = axis == 2 ? INPLACE_ROW_WORDS / nt : words <= (uint32_t)nt ? 1 : words <= 2u * nt ? 2 : 4;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3((unsigned)nt);
    cfg.dynamicSmemBytes = (smem_words(axis, nw * nt) + P.T.S1 + (P.thr_smem ? P.T.NC * P.T.NC * P.T.S1 : 0u)) * 4;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {const_cast<InplaceParams*>(&P)};
    CS_CUDA(cudaLaunchKernelExC(&cfg, kernel_of(K, axis, nw), args));
}

static dim3 pack_grid(uint32_t n_rep) {
    const uint32_t y = n_rep < 32768u ? n_rep : 32768u;
    return dim3(y >= 2048u ? 1u : 2048u / y, y);
}

void inplace_pack(int K, const InplaceParams& P, cudaStream_t s) {
    if (K == 16) inplace_pack_kernel<16><<<pack_grid(P.n_rep), 256, 0, s>>>(P);
    else inplace_pack_kernel<8><<<pack_grid(P.n_rep), 256, 0, s>>>(P);
    CS_LAUNCH_CHECK();
}

void inplace_unpack(int K, const InplaceParams& P, cudaStream_t s) {
    if (K == 16) inplace_unpack_kernel<16><<<pack_grid(P.n_rep), 256, 0, s>>>(P);
    else inplace_unpack_kernel<8><<<pack_grid(P.n_rep), 256, 0, s>>>(P);
    CS_LAUNCH_CHECK();
}

void region_windows(const uint8_t* rpad, const RepDesc& rd, uint8_t* wcode, uint32_t* uni, cudaStream_t s) {
    region_window_kernel<<<2048, 256, 0, s>>>(rpad, rd, wcode, uni);
    CS_LAUNCH_CHECK();
}

void inplace_view(int K, const InplaceParams& P, const RepDesc& rd, uint32_t num_sms, float* out, cudaStream_t s) {
    const uint64_t words = (uint64_t)rd.X * rd.Y * rd.Wz;
    // words of a warp (at most 32, one per lane): few enough that small lattices still fill the chip
    const uint64_t most = words / (num_sms * 32u) + 1u;
    const uint32_t per = most < 32u ? (uint32_t)most : 32u;
    const uint64_t blocks = (words + 8u * per - 1u) / (8u * per);
    const unsigned grid = (unsigned)(blocks < 4096u ? blocks : 4096u);
    if (K == 16) inplace_view_kernel<16><<<grid, 256, 0, s>>>(P, rd, out, per);
    else inplace_view_kernel<8><<<grid, 256, 0, s>>>(P, rd, out, per);
    CS_LAUNCH_CHECK();
}

}  // namespace cellsim
