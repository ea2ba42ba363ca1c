// device_lists.cu — the list form of the production step (see lists_kernel.cuh).
#include <cuda_runtime.h>

#include "cuda_check.h"
#include "lists_kernel.cuh"
#include "prod_kernel.cuh"
#include "views.cuh"

namespace cellsim {

namespace {

constexpr uint32_t EMPTY = 0xFFFFFFFFu;  // free hash slot (no voxel packs to it)
constexpr uint32_t NONE = 0xFFFFu;       // no entry

// Byte offsets of a block's shared-memory areas.  Per entry: content, new content, Philox block B(v, 0),
// voxel, move mask, the hash slots of its targets, its own slot, the frame of its Philox block, whether the
// new content holds.  Per hash slot (two per entry): voxel, entry, movers from below and above.
struct ListLayout {
    size_t c, nc, b, xyz, d, out, key, sl, slot, bf, hv, tch, pend, thr, cnt, total;
};
__host__ __device__ inline size_t list_take(size_t& o, size_t bytes) {
    const size_t at = o;
    o += (bytes + 15u) & ~(size_t)15u;
    return at;
}
__host__ __device__ inline ListLayout list_layout(int K, uint32_t cap, uint32_t thr_words) {
    ListLayout L;
    size_t o = 0;
    const uint32_t hs = 2u * cap;
    L.c = list_take(o, (size_t)K * cap);
    L.nc = list_take(o, (size_t)K * cap);
    L.b = list_take(o, 16u * (size_t)cap);
    L.xyz = list_take(o, 4u * (size_t)cap);
    L.d = list_take(o, 4u * (size_t)cap);
    L.out = list_take(o, 4u * (size_t)cap);
    L.key = list_take(o, 4u * (size_t)hs);
    L.sl = list_take(o, 4u * (size_t)hs);
    L.hv = list_take(o, 2u * (size_t)hs);
    L.slot = list_take(o, 2u * (size_t)cap);
    L.bf = list_take(o, 2u * (size_t)cap);
    L.tch = list_take(o, (size_t)cap);
    L.pend = list_take(o, 2u * (size_t)cap);
    L.thr = list_take(o, 4u * (size_t)thr_words);
    L.cnt = list_take(o, 4u * (16 + PD_N));
    L.total = o;
    return L;
}

template <int K>
__device__ __forceinline__ Vox<K> ls_load(const uint8_t* p) {
    Vox<K> c;
    if constexpr (K == 16) {
        const uint4 t = *reinterpret_cast<const uint4*>(p);
        c.w[0] = (uint64_t)t.x | ((uint64_t)t.y << 32);
        c.w[1] = (uint64_t)t.z | ((uint64_t)t.w << 32);
    } else {
        const uint2 t = *reinterpret_cast<const uint2*>(p);
        c.w[0] = (uint64_t)t.x | ((uint64_t)t.y << 32);
    }
    return c;
}

struct Rep {
    RepDesc rd;
    uint32_t code;  // uniform region code or 0
    const uint8_t* rpad;
    const uint32_t* thr;
    uint32_t S1, NC;
};

// Region code of voxel (x, y, z); 0 outside the lattice.
__device__ __forceinline__ uint32_t code_at(const Rep& R, uint32_t x, uint32_t y, uint32_t z) {
    if (x >= R.rd.X || y >= R.rd.Y || z >= R.rd.Z) return 0u;  // -1 wraps to a large number
    if (R.code) return R.code;
    return __ldg(R.rpad + ((uint64_t)x * R.rd.Y + y) * R.rd.Zr + z + 2u);
}

// Move mask (as decide_moves) of a voxel for one sweep, w0 = B(v, 0)[sweep].
template <int K>
__device__ __forceinline__ uint32_t moves_along(const Rep& R, const Vox<K>& c, uint32_t x, uint32_t y, uint32_t z,
                                                uint32_t v, uint32_t frame, uint32_t sweep, uint32_t w0) {
    const uint32_t dx = sweep == 0u, dy = sweep == 1u, dz = sweep == 2u;
    const uint32_t rs = code_at(R, x, y, z) * R.NC;
    const uint32_t* tlo = R.thr + (rs + code_at(R, x - dx, y - dy, z - dz)) * R.S1;
    const uint32_t* thi = R.thr + (rs + code_at(R, x + dx, y + dy, z + dz)) * R.S1;
    return decide_moves<K>(c, v, frame, sweep, tlo, thi, R.rd.seed_lo, R.rd.seed_hi, w0);
}

template <int K>
__device__ __forceinline__ bool list_calm(const ProdTables& T, uint32_t ci, const Vox<K>& c, uint32_t w3) {
    return calm_voxel<K>(c, w3, T.quiet + (size_t)ci * T.S1 * T.QS, T.QS, T.one + (size_t)ci * T.S1 * 3, T.g23 + 2 * ci,
                         T.a2 ? T.a2 + (size_t)ci * T.S1 * T.S1 : nullptr, T.tau);
}

template <int K, int NT>
__global__ void __launch_bounds__(NT, NT > 256 ? 1 : 2) list_frames_kernel(const __grid_constant__ ListParams P) {
    extern __shared__ __align__(16) unsigned char sm[];
    const uint32_t cap = P.cap, HS = 2u * cap;
    const ListLayout L = list_layout(K, cap, P.thr_words);
    Vox<K>* const c = reinterpret_cast<Vox<K>*>(sm + L.c);
    Vox<K>* const nc = reinterpret_cast<Vox<K>*>(sm + L.nc);
    uint4* const b = reinterpret_cast<uint4*>(sm + L.b);
    uint32_t* const xyz = reinterpret_cast<uint32_t*>(sm + L.xyz);
    uint32_t* const d = reinterpret_cast<uint32_t*>(sm + L.d);
    ushort2* const out = reinterpret_cast<ushort2*>(sm + L.out);    // slots of the targets below / above
    uint32_t* const key = reinterpret_cast<uint32_t*>(sm + L.key);
    ushort2* const sl = reinterpret_cast<ushort2*>(sm + L.sl);      // entries moving in from below / above
    uint16_t* const hv = reinterpret_cast<uint16_t*>(sm + L.hv);
    uint16_t* const slot = reinterpret_cast<uint16_t*>(sm + L.slot);
    uint16_t* const bf = reinterpret_cast<uint16_t*>(sm + L.bf);
    uint8_t* const tch = sm + L.tch;
    uint16_t* const pend = reinterpret_cast<uint16_t*>(sm + L.pend);
    // cnt[0]: entries, cnt[1]: compacted entries, cnt[2 + (f & 1)]: voxels that may react, cnt[4]: particles
    uint32_t* const cnt = reinterpret_cast<uint32_t*>(sm + L.cnt);
    uint32_t* const s_diag = cnt + 16;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t rep = P.rep0 + blockIdx.x;
    Rep R;
    R.rd = P.reps[rep];
    R.code = (R.rd.flags & 1u) ? 1u : P.code;
    R.rpad = P.region_pad + R.rd.rbase;
    R.S1 = P.T.S1;
    R.NC = P.T.NC;
    R.thr = P.T.thr;
    const uint32_t ci = R.rd.counts_index;
    const uint32_t Y = R.rd.Y, Z = R.rd.Z, k0 = R.rd.seed_lo, k1 = R.rd.seed_hi;
    if (P.thr_words) {
        uint32_t* const s_thr = reinterpret_cast<uint32_t*>(sm + L.thr);
        for (uint32_t i = tid; i < P.thr_words; i += NT) s_thr[i] = P.T.thr[i];
        R.thr = s_thr;
    }
    if (tid < 16 + PD_N) cnt[tid] = 0u;
    if (blockIdx.x == 0 && tid == 0) *P.step_out = P.frame0 + P.n_frames;
    const uint32_t n_in = P.n[rep];
    const uint64_t gl = (uint64_t)rep * cap;
    auto clear_hash = [&]() {
        for (uint32_t i = tid; i < HS; i += NT) {
            key[i] = EMPTY;
            sl[i] = make_ushort2((unsigned short)NONE, (unsigned short)NONE);
        }
    };
    // the slot of voxel t, taken if it had none (fresh); HS is twice the entries, so a free slot is found
    auto find = [&](uint32_t t, bool& fresh) -> uint32_t {
        uint32_t s = __umulhi(t * 0x9E3779B1u, HS);
        for (uint32_t tries = 0; tries < HS; tries++) {
            const uint32_t old = atomicCAS(&key[s], EMPTY, t);
            if (old == EMPTY || old == t) {
                fresh = old == EMPTY;
                return s;
            }
            s = s + 1u == HS ? 0u : s + 1u;
        }
        fresh = false;
        return 0u;
    };
    auto voxel = [&](uint32_t t) -> uint32_t { return ((t >> 20) * Y + ((t >> 10) & 1023u)) * Z + (t & 1023u); };
    if (n_in & LIST_STOPPED) return;
    clear_hash();
    __syncthreads();
    uint32_t np = 0u;
    for (uint32_t i = tid; i < n_in; i += NT) {
        const uint32_t t = P.xyz[gl + i];
        const Vox<K> w = ls_load<K>(P.cont + (gl + i) * K);
        bool fresh;
        const uint32_t s = find(t, fresh);
        xyz[i] = t;
        c[i] = w;
        slot[i] = (uint16_t)s;
        hv[s] = (uint16_t)i;
        tch[i] = 0u;
        bf[i] = (uint16_t)(P.frame0 - 1u);
        np += vox_n<K>(w);
    }
    np = __reduce_add_sync(0xffffffffu, np);
    if (lane == 0u && np) atomicAdd(&cnt[4], np);
    if (tid == 0u) cnt[0] = n_in;
    __syncthreads();

    // B(v, 0) of entry i in frame fr, evaluated on its first use in the frame
    auto block0 = [&](uint32_t i, uint32_t v, uint32_t fr) -> uint4 {
        if (bf[i] == (uint16_t)fr) return b[i];
        const U4 u = d_philox(v, fr, 0u, 0u, k0, k1);
        const uint4 w = make_uint4(u.x, u.y, u.z, u.w);
        b[i] = w;
        bf[i] = (uint16_t)fr;
        return w;
    };
    uint32_t n = n_in;  // entries; the same value in every thread
    // The occupied entries to the front of the list, the hash made anew.
    auto compact = [&](uint32_t fr) {
        for (uint32_t i = tid; i < n; i += NT)
            if (tch[i]) c[i] = nc[i];
        if (tid == 0u) cnt[1] = 0u;
        __syncthreads();
        for (uint32_t i = tid; i < n; i += NT) {
            const Vox<K> w = c[i];
            if (vox_empty<K>(w)) continue;
            const uint32_t p = atomicAdd(&cnt[1], 1u);
            nc[p] = w;
            d[p] = xyz[i];
        }
        clear_hash();
        __syncthreads();
        n = cnt[1];
        for (uint32_t i = tid; i < n; i += NT) {
            const uint32_t t = d[i];
            bool fresh;
            const uint32_t s = find(t, fresh);
            c[i] = nc[i];
            xyz[i] = t;
            slot[i] = (uint16_t)s;
            hv[s] = (uint16_t)i;
            tch[i] = 0u;
            bf[i] = (uint16_t)(fr - 1u);
        }
        if (tid == 0u) cnt[0] = n;
        __syncthreads();
    };

    const uint32_t* const rowu = R.thr + (R.code * R.NC + R.code) * R.S1;
    uint32_t f = 0;
    for (; f < P.n_frames; f++) {
        const uint32_t fr = P.frame0 + f;
        if (2u * cnt[4] > cap) break;  // the frame might not fit; particles are the same in all its sweeps
        for (uint32_t sweep = 0; sweep < 3u; sweep++) {
            // an axis of length 1 has no neighbour: every decision is 0 and every content stays
            if ((sweep == 0u ? R.rd.X : sweep == 1u ? Y : Z) == 1u) continue;
            // a sweep makes at most one entry per particle
            if (n + cnt[4] > cap) compact(fr);
            const uint32_t stride = sweep == 0u ? Y * Z : sweep == 1u ? Z : 1u;
            const uint32_t shift = sweep == 0u ? 20u : sweep == 1u ? 10u : 0u;
            const uint32_t dim = sweep == 0u ? R.rd.X : sweep == 1u ? Y : Z;
            const uint32_t step = sweep == 0u ? 1u << 20 : sweep == 1u ? 1u << 10 : 1u;
            // 1.
            for (uint32_t i = tid; i < n; i += NT) {
                if (tch[i]) {
                    c[i] = nc[i];
                    tch[i] = 0u;
                }
                const Vox<K> w = c[i];
                uint32_t m = 0u;
                if (!vox_empty<K>(w)) {
                    const uint32_t t = xyz[i], v = voxel(t);
                    const uint4 b0 = block0(i, v, fr);
                    const uint32_t w0 = sweep == 0u ? b0.x : sweep == 1u ? b0.y : b0.z;
                    if (R.code && vox_n<K>(w) == 1u) {
                        // one particle, one region: one threshold, or 0 towards the lattice's faces
                        const uint32_t th = rowu[(uint32_t)w.w[0]], at = (t >> shift) & 1023u;
                        const uint32_t tm = at > 0u ? th : 0u, tp = at + 1u < dim ? th : 0u;
                        m = w0 < tm ? 1u : w0 - tm < tp ? 0x10000u : 0u;
                    } else {
                        m = moves_along<K>(R, w, t >> 20, (t >> 10) & 1023u, t & 1023u, v, fr, sweep, w0);
                    }
#pragma unroll 1
                    for (uint32_t up = 0; up < 2u; up++) {
                        if (((m >> (16u * up)) & 0xFFFFu) == 0u) continue;
                        const uint32_t tt = up ? t + step : t - step;
                        bool fresh;
                        const uint32_t s = find(tt, fresh);
                        if (fresh) {
                            const uint32_t j = atomicAdd(&cnt[0], 1u);
                            xyz[j] = tt;
                            c[j] = vox_zero<K>();
                            d[j] = 0u;
                            tch[j] = 0u;
                            slot[j] = (uint16_t)s;
                            bf[j] = (uint16_t)(fr - 1u);
                            hv[s] = (uint16_t)j;
                        }
                        if (up) {
                            sl[s].x = (uint16_t)i;
                            out[i].y = (uint16_t)s;
                        } else {
                            sl[s].y = (uint16_t)i;
                            out[i].x = (uint16_t)s;
                        }
                    }
                }
                d[i] = m;
            }
            __syncthreads();
            // 2.
            n = cnt[0];
            for (uint32_t i = tid; i < n; i += NT) {
                const uint32_t m = d[i], s = slot[i];
                const ushort2 in = sl[s];
                if (m == 0u && in.x == NONE && in.y == NONE) continue;
                sl[s] = make_ushort2((unsigned short)NONE, (unsigned short)NONE);
                Vox<K> lo = vox_zero<K>(), hi = vox_zero<K>();
                uint32_t dlo = 0u, dhi = 0u;
                if (in.x != NONE) {
                    lo = c[in.x];
                    dlo = d[in.x];
                } else if (m & 0xFFFFu) {
                    lo = c[hv[out[i].x]];
                }
                if (in.y != NONE) {
                    hi = c[in.y];
                    dhi = d[in.y];
                } else if (m >> 16) {
                    hi = c[hv[out[i].y]];
                }
                const uint32_t v = voxel(xyz[i]);
                nc[i] = combine<K>(c[i], m, lo, dlo, hi, dhi, v, v - stride, v + stride, fr, sweep);
                tch[i] = 1u;
            }
            __syncthreads();
        }
        // reactions
        uint32_t* const n_pend = &cnt[2u + (f & 1u)];
        if (tid == 0u) cnt[2u + ((f & 1u) ^ 1u)] = 0u;
        for (uint32_t i = tid; i < n; i += NT) {
            if (tch[i]) {
                c[i] = nc[i];
                tch[i] = 0u;
            }
            const Vox<K> w = c[i];
            if (vox_empty<K>(w)) continue;
            const uint4 b0 = block0(i, voxel(xyz[i]), fr);
            if (!list_calm<K>(P.T, ci, w, b0.w)) pend[atomicAdd(n_pend, 1u)] = (uint16_t)i;
        }
        __syncthreads();
        const uint32_t m = *n_pend;
        if (m) {
                for (uint32_t q = warp; q < m; q += NT / 32) {
                    const uint32_t i = pend[q], v = voxel(xyz[i]);
                    Vox<K> r = c[i];
                    const uint32_t n0 = vox_n<K>(r), w3 = b[i].w;
                    const bool fired = react_voxel_warp<K>(r, 0u, v, fr, k0, k1, R.rd.rate_mult, P.T, nullptr,
                                                           P.counts + (size_t)ci * R.S1, s_diag, w3);
                    __syncwarp();
                    if (lane == 0u && fired) {
                        c[i] = r;
                        atomicAdd(&cnt[4], vox_n<K>(r) - n0);
                    }
                    __syncwarp();
                }
            __syncthreads();
        }
        // emptied entries out while no Philox block is lost; the sweeps make sure of the room
        if (f + 1u < P.n_frames && 2u * n > 3u * cnt[4]) compact(fr);
    }
    __syncthreads();
    if (tid == 0u) cnt[1] = 0u;
    __syncthreads();
    for (uint32_t i = tid; i < n; i += NT) {
        const Vox<K> w = c[i];
        if (vox_empty<K>(w)) continue;
        const uint32_t p = atomicAdd(&cnt[1], 1u);
        P.xyz[gl + p] = xyz[i];
        st_vox_g<K>(P.cont + (gl + p) * K, w);
    }
    __syncthreads();
    if (tid == 0u) {
        const bool stopped = f < P.n_frames;
        P.n[rep] = stopped ? cnt[1] | LIST_STOPPED : cnt[1];
        if (stopped) {
            P.at[rep] = P.frame0 + f;
            *P.host_flag = 1u;
        }
    }
    if (tid < PD_N && s_diag[tid]) atomicAdd(P.diag + tid, s_diag[tid]);
}

// Appends the occupied voxels of every replicate's slots to its list (blockIdx.y: replicates).
template <int K>
__global__ void __launch_bounds__(256) list_pack_kernel(const ListParams P, uint32_t n_rep) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t rep = blockIdx.y; rep < n_rep; rep += gridDim.y) {
        const RepDesc rd = P.reps[rep];
        const uint32_t V = rd.X * rd.Y * rd.Z;
        const uint64_t gl = (uint64_t)rep * P.cap;
        for (uint64_t base = ((uint64_t)blockIdx.x * 256u + threadIdx.x) & ~31ull; base < V;
             base += (uint64_t)gridDim.x * 256u) {
            const uint32_t v = (uint32_t)base + lane;
            Vox<K> c = vox_zero<K>();
            if (v < V) c = ls_load<K>(P.lat + (rd.base + v) * K);
            const bool occupied = !vox_empty<K>(c);
            const uint32_t m = __ballot_sync(0xffffffffu, occupied);
            if (m == 0u) continue;
            uint32_t at = 0u;
            if (lane == 0u) at = atomicAdd(P.n + rep, (uint32_t)__popc(m));
            at = __shfl_sync(0xffffffffu, at, 0) + (uint32_t)__popc(m & ((1u << lane) - 1u));
            if (occupied && at < P.cap) {
                const uint32_t xy = v / rd.Z, z = v - xy * rd.Z, x = xy / rd.Y;
                P.xyz[gl + at] = x << 20 | (xy - x * rd.Y) << 10 | z;
                st_vox_g<K>(P.cont + (gl + at) * K, c);
            }
        }
    }
}

// A replicate with more occupied voxels than its list holds keeps its state in the slots.
__global__ void list_check_kernel(const ListParams P, uint32_t n_rep) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n_rep && P.n[r] > P.cap) {
        P.n[r] = LIST_DENSE;
        P.at[r] = P.frame0;
        *P.host_flag = 1u;
    }
}

// Zeros in the slots of every replicate whose state is its list.
template <int K>
__global__ void __launch_bounds__(256) list_zero_kernel(const ListParams P, uint32_t n_rep) {
    for (uint32_t rep = blockIdx.y; rep < n_rep; rep += gridDim.y) {
        if (P.n[rep] == LIST_DENSE) continue;
        const RepDesc rd = P.reps[rep];
        const uint32_t V = rd.X * rd.Y * rd.Z;
        for (uint64_t v = (uint64_t)blockIdx.x * 256u + threadIdx.x; v < V; v += (uint64_t)gridDim.x * 256u)
            st_vox_g<K>(P.lat + (rd.base + v) * K, vox_zero<K>());
    }
}

// Writes the lists into the zeroed slots.
template <int K>
__global__ void __launch_bounds__(256) list_unpack_kernel(const ListParams P, uint32_t n_rep) {
    for (uint32_t rep = blockIdx.y; rep < n_rep; rep += gridDim.y) {
        if (P.n[rep] == LIST_DENSE) continue;
        const uint32_t n = P.n[rep] & ~LIST_STOPPED;
        const RepDesc rd = P.reps[rep];
        const uint64_t gl = (uint64_t)rep * P.cap;
        for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u) {
            const uint32_t t = P.xyz[gl + i];
            const uint32_t v = ((t >> 20) * rd.Y + ((t >> 10) & 1023u)) * rd.Z + (t & 1023u);
            st_vox_g<K>(P.lat + (rd.base + v) * K, ls_load<K>(P.cont + (gl + i) * K));
        }
    }
}

// View 0 (views.cuh) of replicate 0 into zeroed floats, from its list.
template <int K>
__global__ void __launch_bounds__(256) list_view_kernel(const ListParams P, float* out) {
    const RepDesc rd = P.reps[0];
    const uint32_t n = P.n[0] == LIST_DENSE ? 0u : P.n[0] & ~LIST_STOPPED;
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u) {
        const uint32_t t = P.xyz[i];
        out[((t >> 20) * rd.Y + ((t >> 10) & 1023u)) * rd.Z + (t & 1023u)] =
            __fdiv_rn((float)view_majority<K>(ls_load<K>(P.cont + (uint64_t)i * K).w), 255.0f);
    }
}

}  // namespace

size_t lists_smem(int K, uint32_t cap, uint32_t thr_words) { return list_layout(K, cap, thr_words).total; }

void lists_set_attrs(int device) {
    int optin = 0;
    CS_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    void* fns[] = {reinterpret_cast<void*>(&list_frames_kernel<8, 256>), reinterpret_cast<void*>(&list_frames_kernel<8, 512>),
                   reinterpret_cast<void*>(&list_frames_kernel<8, 768>), reinterpret_cast<void*>(&list_frames_kernel<16, 256>),
                   reinterpret_cast<void*>(&list_frames_kernel<16, 512>), reinterpret_cast<void*>(&list_frames_kernel<16, 768>)};
    for (void* fn : fns) {
        CS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
        CS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    }
}

void lists_launch(int K, int threads, const ListParams& P, uint32_t grid, cudaStream_t s) {
    if (grid == 0 || P.n_frames == 0) return;
    const size_t smem = lists_smem(K, P.cap, P.thr_words);
    auto run = [&](auto kernel) { kernel<<<grid, threads, smem, s>>>(P); };
    if (K == 16) run(threads == 768 ? list_frames_kernel<16, 768> : threads == 512 ? list_frames_kernel<16, 512> : list_frames_kernel<16, 256>);
    else run(threads == 768 ? list_frames_kernel<8, 768> : threads == 512 ? list_frames_kernel<8, 512> : list_frames_kernel<8, 256>);
    CS_LAUNCH_CHECK();
}

// Blocks of a launch over all replicates: x over a replicate's voxels, y over the replicates.
static dim3 rep_grid(uint64_t voxels_max, uint32_t n_rep) {
    const uint32_t y = n_rep < 32768u ? n_rep : 32768u;
    const uint64_t x = (voxels_max + 255u) / 256u, most = y >= 2048u ? 1u : 2048u / y;
    return dim3((unsigned)(x < most ? x : most), y);
}

void lists_pack(int K, const ListParams& P, uint32_t n_rep, uint64_t voxels_max, cudaStream_t s) {
    CS_CUDA(cudaMemsetAsync(P.n, 0, (size_t)n_rep * 4, s));
    const dim3 g = rep_grid(voxels_max, n_rep);
    if (K == 16) list_pack_kernel<16><<<g, 256, 0, s>>>(P, n_rep);
    else list_pack_kernel<8><<<g, 256, 0, s>>>(P, n_rep);
    CS_LAUNCH_CHECK();
    list_check_kernel<<<(n_rep + 255u) / 256u, 256, 0, s>>>(P, n_rep);
    CS_LAUNCH_CHECK();
}

void lists_unpack(int K, const ListParams& P, uint32_t n_rep, uint64_t voxels_max, cudaStream_t s) {
    const dim3 g = rep_grid(voxels_max, n_rep), gu(4u, g.y);
    if (K == 16) {
        list_zero_kernel<16><<<g, 256, 0, s>>>(P, n_rep);
        list_unpack_kernel<16><<<gu, 256, 0, s>>>(P, n_rep);
    } else {
        list_zero_kernel<8><<<g, 256, 0, s>>>(P, n_rep);
        list_unpack_kernel<8><<<gu, 256, 0, s>>>(P, n_rep);
    }
    CS_LAUNCH_CHECK();
}

void lists_view(int K, const ListParams& P, const RepDesc& rd, float* out, cudaStream_t s) {
    CS_CUDA(cudaMemsetAsync(out, 0, (size_t)rd.X * rd.Y * rd.Z * sizeof(float), s));
    if (K == 16) list_view_kernel<16><<<16, 256, 0, s>>>(P, out);
    else list_view_kernel<8><<<16, 256, 0, s>>>(P, out);
    CS_LAUNCH_CHECK();
}

}  // namespace cellsim
