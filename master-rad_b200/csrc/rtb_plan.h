// Host arithmetic of the frame and replay launches: items, path slots, grids and the bytes of
// their buffers.  No CUDA in it, so that a test can compile it for the host and walk its sizes.
#pragma once
#include <algorithm>
#include <cstddef>

namespace rtb {

constexpr int kBlock = 1024, kSmallBlock = 128;  // of the two forms, see rtb_paths.cuh
constexpr int kSlotsPerLane = 6;   // 4: 5 % slower (more phases), 8: 2 % (the slots leave L2)
constexpr int kGroupBytes = 32 * 96;  // 32 path slots, see Slot

// A block's slots and the two lists that name them.
inline size_t block_path_bytes(int slots) {
  return (size_t)((slots + 31) / 32) * (kGroupBytes + 2 * 32 * sizeof(int));
}

// Lanes of each warp that take one of n rays or items.  Few go to few lanes of many warps: a
// warp walks on until the longest of its rays ends and runs every branch any of them takes, so
// work for less than 32 lanes in kFewWarpsPerSm warps of every SM waits least when it is spread
// over those.  257 rays among 4,096 primitives 67 -> 42 us, 64x36 pixels of 10k primitives 204 ->
// 128 us, of 65 spheres 48 -> 42 us; with 2 / 4 / 16 warps an SM the second takes 164 / 149 / 129,
// the third 46 / 43 / 45.
constexpr int kFewWarpsPerSm = 8;
inline int lanes_per_warp(long long n, int sm_count) {
  const long long warps = (long long)sm_count * kFewWarpsPerSm;
  return (int)std::min<long long>(32, std::max<long long>(1, (n + warps - 1) / warps));
}

// Path slots of each of `blocks` blocks for `items`: `most` on large frames; where the items
// fill them only a few times, the number that divides them into equal rounds (a last round of a
// few slots costs nearly a whole one).  More items may need fewer slots: one round more.
inline int slots_in_rounds(long long items, long long blocks, long long most) {
  const long long rounds = (items + blocks * most - 1) / (blocks * most);
  return (int)std::min(most, std::max<long long>(32, (items + blocks * rounds - 1) / (blocks * rounds)));
}

// How a frame's pixels become queue items and a launch.
struct FrameShape {
  int block = 0;              // kBlock: k_render, kSmallBlock: k_render_small
  int sm_count = 0;
  int spp = 1;
  long long pixels = 0;
  long long resident = 0;     // threads of a full-occupancy grid
  long long tail_pixels = 0;  // the frame's last pixels, queued one sample per item
  // by set_tail
  long long split = 0, items = 0, grid = 0;
  int slots = 0;              // path slots a block uses; k_render_small: lanes a warp uses

  void set_tail(long long pixels_in_tail) {
    tail_pixels = pixels_in_tail;
    split = pixels - tail_pixels;
    items = split + tail_pixels * spp;
    const long long blocks = resident / block;
    long long per_block;
    if (block == kSmallBlock) {
      slots = lanes_per_warp(items, sm_count);
      per_block = (long long)slots * (kSmallBlock / 32);
    } else {
      slots = slots_in_rounds(items, blocks, kSlotsPerLane * kBlock);
      per_block = slots;
    }
    grid = std::min(blocks, (items + per_block - 1) / per_block);
  }
  // In k_render_small's form; the tail stays as long as it was.
  void without_slots(long long small_resident) {
    block = kSmallBlock;
    resident = small_resident;
    set_tail(tail_pixels);
  }
  size_t tail_bytes() const { return (size_t)tail_pixels * spp * 3 * sizeof(float); }
  size_t path_bytes() const { return block == kBlock ? (size_t)grid * block_path_bytes(slots) : 0; }
};

// Settles a frame's buffers: grow_tail(bytes) and grow_paths(bytes) say whether the buffer is
// there.  Without a sample buffer every pixel keeps its samples in one slot; without path slots
// the frame runs in the form that needs none, of small_resident() threads.  The slots are asked
// for last: their number depends on the tail, and does not only shrink without it.
template <class Tail, class Paths, class Small>
inline void settle_frame(FrameShape& f, Tail&& grow_tail, Paths&& grow_paths, Small&& small_resident) {
  if (!grow_tail(f.tail_bytes())) f.set_tail(0);
  if (f.block == kBlock && !grow_paths(f.path_bytes())) f.without_slots(small_resident());
}

// The path slots of a replay in phases, one block an SM: as a frame's, but vertices of
// kMaxVertexBytes at most.
constexpr long long kMaxVertexBytes = 256LL << 20;
struct ReplayShape {
  long long grid = 0;
  int slots = 0;
  size_t path_bytes = 0, vertex_bytes = 0;  // the vertices lie behind the slots
  ReplayShape(long long samples, int max_depth, int sm_count) : grid(sm_count) {
    const long long vertex = 2LL * 16 * max_depth;  // two float4 a segment
    const long long most = std::max<long long>(
        kBlock, std::min<long long>(kSlotsPerLane * kBlock, kMaxVertexBytes / (vertex * grid) / kBlock * kBlock));
    slots = slots_in_rounds(samples, grid, most);
    path_bytes = ((size_t)grid * block_path_bytes(slots) + 255) & ~(size_t)255;
    vertex_bytes = (size_t)(grid * slots * vertex);
  }
};

}  // namespace rtb
