// views.cuh — the headless visualisation views of final_stage.wgsl:35-68,
// written to a float volume in lattice order instead of a storage texture.
//
//   view 0  majority species of the voxel's slots / 255 (the first slot whose
//           species count is strictly largest wins, final_stage.wgsl:43-57)
//   view 1  region id / 255 (final_stage.wgsl:60-62)
//   view 2  reservoir species / 255 (final_stage.wgsl:64-66)
//
// Voxels cut away by the slice, res[axis] - coord[axis] < slice
// (final_stage.wgsl:35-38), are 0.
#pragma once
#include <cstdint>

namespace cellsim {

struct ViewParams {
    const uint8_t* slots;      // [V][K], compacted
    uint32_t K;
    uint32_t X, Y, Z;
    const uint8_t* region_id;  // [V] region ids, or null
    const uint8_t* region_pad; // padded region codes (id + 1), rows of Zr bytes with z at column z + 2, or null
    uint32_t Zr;
    const uint8_t* reservoir;  // [V], or null (no reservoirs)
    int32_t view;
    int32_t slice_axis;
    uint32_t slice;
    float* out;                // [V]
};

static __global__ void render_view_kernel(ViewParams p) {
    const uint64_t V = (uint64_t)p.X * p.Y * p.Z;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t z = (uint32_t)(v % p.Z);
        const uint64_t xy = v / p.Z;
        const uint32_t y = (uint32_t)(xy % p.Y), x = (uint32_t)(xy / p.Y);
        const uint32_t res[3] = {p.X, p.Y, p.Z}, coord[3] = {x, y, z};
        const int a = p.slice_axis < 0 || p.slice_axis > 2 ? 0 : p.slice_axis;
        if (res[a] - coord[a] < p.slice) {
            p.out[v] = 0.0f;
            continue;
        }
        uint32_t value = 0;
        if (p.view == 1) {
            if (p.region_id) value = p.region_id[v];
            else if (p.region_pad) value = (uint32_t)p.region_pad[xy * p.Zr + z + 2] - 1u;
        } else if (p.view == 2) {
            value = p.reservoir ? p.reservoir[v] : 0u;
        } else {
            const uint8_t* s = p.slots + v * p.K;
            uint32_t n = 0;
            while (n < p.K && s[n]) n++;
            uint32_t best = 0;
            for (uint32_t i = 0; i < n; i++) {
                uint32_t c = 0;
                for (uint32_t j = 0; j < n; j++) c += s[i] == s[j];
                if (c > best) {
                    best = c;
                    value = s[i];
                }
            }
        }
        p.out[v] = __fdiv_rn((float)value, 255.0f);
    }
}

// The majority species of K slot bytes held in 64-bit words (byte i of the words = slot i), as above:
// the occupied slots end at the first empty one.
template <int K>
__device__ __forceinline__ uint32_t view_majority(const uint64_t (&w)[K / 8]) {
    auto slot = [&](uint32_t i) -> uint32_t { return (uint32_t)((K == 8 || i < 8u ? w[0] : w[K / 8 - 1]) >> (8u * (i & 7u))) & 0xFFu; };
    uint32_t n = 0;
    while (n < (uint32_t)K && slot(n)) n++;
    uint32_t value = n ? slot(0) : 0u, best = 0;  // one or two particles: the first slot's species
    if (n > 2u)
        for (uint32_t i = 0; i < n; i++) {
            uint32_t c = 0;
            for (uint32_t j = 0; j < n; j++) c += slot(i) == slot(j);
            if (c > best) {
                best = c;
                value = slot(i);
            }
        }
    return value;
}

// View 0 of the whole volume (no slice) from K = 8 or 16 slots per voxel: one vector load and one
// coalesced store per voxel and no coordinates, so that it runs at the copy bandwidth (256^3, K = 16: 320
// MB; a call that ends in one view takes 64 us less than with render_view_kernel's division chain and byte
// loads per voxel, which took 135 us).
template <int K>
static __global__ void __launch_bounds__(256) majority_view_kernel(const uint8_t* slots, uint64_t V, float* out) {
    for (uint64_t v = (uint64_t)blockIdx.x * 256u + threadIdx.x; v < V; v += (uint64_t)gridDim.x * 256u) {
        uint64_t w[K / 8];
        if constexpr (K == 16) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(slots + v * 16u);
            w[0] = t.x;
            w[1] = t.y;
        } else {
            w[0] = *reinterpret_cast<const uint64_t*>(slots + v * 8u);
        }
        out[v] = __fdiv_rn((float)((w[0] & 0xFFull) == 0ull ? 0u : view_majority<K>(w)), 255.0f);
    }
}

static void launch_majority_view(uint32_t K, const uint8_t* slots, uint64_t V, float* out, cudaStream_t s) {
    const unsigned grid = (unsigned)(V < 256u * 8192u ? (V + 255u) / 256u : 8192u);
    if (K == 16) majority_view_kernel<16><<<grid, 256, 0, s>>>(slots, V, out);
    else majority_view_kernel<8><<<grid, 256, 0, s>>>(slots, V, out);
}

}  // namespace cellsim
