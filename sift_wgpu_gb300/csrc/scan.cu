// scan.cu — the oriented list, in the reference's (keypoint, bin) order.
//
// Candidate slot i holds c_i peaks (0 if refinement or the orientation stage
// rejected it) and writes its c_i oriented copies at the sum of the counts
// before it: the counts of the tiles before its own (kSlotTile slots each,
// counted by the orientation stage), then those before it in its tile. Every
// position is an exact integer sum, so the result does not depend on
// scheduling. (A scan kernel of its own ahead of this one took 7.7 us of a
// 1080p frame's octave-0 chain, of which 5 us are left.)
#include <algorithm>

#include "tile_scan.cuh"

namespace sift {
namespace {

// Octave o's oriented keypoints go after those of octaves 0..o-1 (whose
// counts are final: their launches of this kernel precede this one). ori_off,
// where not null, receives each slot's first output position in the octave.
// (The count is the sum of the tiles: an atomic per warp of the orientation
// stage on the word beside its work queue's took that stage from 41 to 48 us.)
__global__ void __launch_bounds__(kSlotTile) k_orient_emit(const Keypoint* __restrict__ refined_at, uint32_t ncap, int o,
                                                           Counters* __restrict__ ctr,
                                                           const float* __restrict__ ori_angle,
                                                           const uint32_t* __restrict__ ori_count,
                                                           const uint32_t* __restrict__ tiles,
                                                           uint32_t* __restrict__ ori_off,
                                                           Keypoint* __restrict__ oriented, uint32_t cap) {
    chain_wait();
    __shared__ uint32_t buf[kSlotTile / 32];
    OctCounters* oc = &ctr->oct[o];
    uint32_t base = 0;
    for (int q = 0; q < o; ++q) base += ctr->oct[q].n_ori;
    const uint32_t n = min(oc->n_cand, ncap);
    if (blockIdx.x == 0) {
        const uint32_t n_ori = tiles_sum<kSlotTile>(tiles, 0, (n + kSlotTile - 1) / kSlotTile, buf);
        if (threadIdx.x == 0) {
            oc->n_ori = n_ori;
            oc->out_base = base;
            atomicAdd(&ctr->n_candidates, oc->n_cand);
            atomicAdd(&ctr->n_refined, oc->n_ref);
            atomicMax(&ctr->n_oriented, base + n_ori);
            if (base + n_ori > cap) atomicOr(&ctr->overflow, 4u);
        }
    }
    uint32_t before = 0, from = 0;
    for (uint32_t t = blockIdx.x; (unsigned long long)t * kSlotTile < n; t += gridDim.x) {
        before += tiles_sum<kSlotTile>(tiles, from, t, buf);
        from = t;
        const uint32_t i = t * kSlotTile + threadIdx.x;
        const uint32_t c = i < n ? ori_count[i] : 0u;
        const uint32_t at = before + block_exclusive<kSlotTile>(c, buf);
        if (i < n && ori_off) ori_off[i] = at;
        if (c == 0) continue;
        const uint32_t off = base + at;
        Keypoint k = refined_at[i];
        for (uint32_t j = 0; j < c; ++j) {
            if (off + j >= cap) break;
            k.angle = ori_angle[(size_t)i * kOriMaxPeaks + j];
            oriented[off + j] = k;
        }
    }
}

}  // namespace

int launch_orient_emit(const Keypoint* refined_at, uint32_t ncap, int o, Counters* ctr, const float* ori_angle,
                       const uint32_t* ori_count, const uint32_t* tiles, uint32_t* ori_off, Keypoint* oriented,
                       uint32_t cap, cudaStream_t st) {
    const unsigned grid = (unsigned)std::max<size_t>(std::min<size_t>(slot_tiles(ncap), 152 * 8), 1);
    if (launch_chained(k_orient_emit, grid, kSlotTile, 0, st, refined_at, ncap, o, ctr, ori_angle, ori_count, tiles,
                       ori_off, oriented, cap) != cudaSuccess)
        return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace sift
