// pass_groups.hpp — how many passes of a frame run side by side (host code).
#pragma once

#include <algorithm>
#include <cstdint>

namespace wpbr {

constexpr uint32_t kMaxGroupPasses = 8;

// Passes per group of a frame. A traversal launch ends with a tail in which
// most of its warps have no ray left (1080p full frame: 31 to 41 % of the warp
// slots active over the launch), and a small film never fills the GPU at all,
// so the passes of a group run as concurrent branches and fill one another's
// tails. 1080p x 16 spp, full frame / textured, groups of 1: 19.9 / 14.6 ms;
// 2: 16.0 / 14.1; 4: 15.2 / 13.8; 8: 14.8 / 13.6. A Sampled64 pass also keeps a
// slot of 64-bin samples per pixel until the group's film gather, so those
// groups stop at 4. Passes times pixels are bounded to 2^24: 4.0 GB of state
// (240 bytes a pixel and pass), and 4.5 GB of Sampled64 slots (268 bytes).
inline uint32_t group_passes(uint64_t pixels, uint32_t spp, bool spectral) {
  const uint64_t k = std::max<uint64_t>(1u, (1ull << 24) / pixels);
  return (uint32_t)std::min<uint64_t>({k, spp, spectral ? 4u : kMaxGroupPasses});
}

// At most as many as may be added to the first pass's buffers, pass_bytes
// each, within a quarter of the free device memory: the context keeps them,
// and they are only there for speed. Contexts that share a GPU (eight films of
// 1080p hold 28 GB so) leave room for one another's scenes.
// (Up to kGroupUnasked bytes nobody asks: the question takes 30 us, 5 % of a
// 256 x 256 preview's first frame.)
constexpr uint64_t kGroupUnasked = 64ull << 20;
inline uint32_t group_passes_within(uint32_t k, uint64_t pass_bytes, uint64_t free_bytes) {
  return (uint32_t)std::min<uint64_t>(k, 1 + free_bytes / 4 / pass_bytes);
}

}  // namespace wpbr
