// The shading order's keys: queue entries are grouped by what they will do in
// the shading kernel, so that the threads of a warp mostly take the same
// branches. A counting sort: whoever learns an entry's hit (the closest-hit
// traversal, or the guide's query kernel) writes its key and counts it;
// k_shade_scatter (integrator.cuh) writes the order.
#pragma once

#include "shading.cuh"

namespace ag {

// Bins: a miss; a Dielectric with its Lambertian lobe only; a Dielectric with
// both lobes; a Conductor; plus kShadeGuided for a vertex the guide samples.
constexpr uint32_t kShadeBins = 8;
constexpr uint32_t kShadeGuided = 4;

// What a key is made from, and where keys and counts go (keys == null: no
// shading order).
struct ShadeKeys {
    const uint32_t* triInfo;
    const uint32_t* sphereMaterial;
    const Material* materials;
    uint32_t sphereCount, materialCount;
    uint8_t* keys;     // a byte per queue entry
    uint32_t* counts;  // kShadeBins words, zeroed by the caller
};

AG_D uint32_t shade_key(const ShadeKeys& s, uint32_t prim, bool guided)
{
    if (prim == 0xffffffffu) return 0u;
    uint32_t mid = (prim & kSpherePrim) ? s.sphereMaterial[min(prim & ~kSpherePrim, s.sphereCount - 1u)]
                                        : __ldg(s.triInfo + prim) & kTriMaterialMask;
    if (mid >= s.materialCount) mid = 0;
    const Material& m = s.materials[mid];
    const uint32_t key = m.kind == kMatConductor ? 3u : (m.lobes == 2u ? 2u : 1u);
    return guided ? key | kShadeGuided : key;
}

// Warp-aggregated rank of this lane's entry among the block's entries with the
// same key, added to hist[key] (shared memory). The whole warp calls it
// together; a lane without an entry passes kShadeBins, which is not counted.
AG_D uint32_t bin_rank(uint32_t* hist, uint32_t key)
{
    const uint32_t peers = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if ((int)(threadIdx.x & 31) == leader && key < kShadeBins) base = atomicAdd(hist + key, __popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    return base + __popc(peers & lanemask_lt());
}

}  // namespace ag
