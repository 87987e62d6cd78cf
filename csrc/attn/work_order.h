// Order in which the blocks of an attention launch take (tile, head) pairs.
//
// Under a causal mask the tiles of a head differ in work by a factor of their number, and blocks start in index
// order, so the longest tiles should come first. But blocks in flight should also share heads: they stream the same
// Q and dO (dK/dV kernel) or K and V (dQ, forward), which only stay in L2 while few heads are in flight. Both are
// served by groups of heads: groups one after another, inside a group the tile index is the slow one.
//
// The group has to be large enough that its longest block, started with the group, does not outlast it. With n tiles
// the longest block has n units of work, a head has n (n + 1) / 2, so 148 SMs are busy with m heads for
// m n (n + 1) / 296 units: m >= 296 / (n + 1). Measured with one head at a time / all heads in one group / this rule
// (dK/dV kernel, 32 heads over 8 KV heads, causal, ratio to the forward kernel of the same run): 1.87 / 1.64 / 1.62
// at 8192 tokens (last block alone for a third of the launch), 1.57 / 1.62 / 1.56 at 32768 (Q and dO of all heads
// are 537 MB).
#pragma once

#if defined(__CUDACC__)
#define ZX_WO_FN __host__ __device__ __forceinline__
#else
#define ZX_WO_FN inline
#endif

namespace zx {

struct WorkItem {
  int tile, head;
};

// Block `bid` of a grid of n_tiles * n_heads; tile 0 of a head comes first.
ZX_WO_FN WorkItem work_item(int bid, int n_tiles, int n_heads, int per_group) {
  const int g = bid / (n_tiles * per_group);
  const int r = bid - g * n_tiles * per_group;
  const int left = n_heads - g * per_group;
  const int size = left < per_group ? left : per_group;
  WorkItem w;
  w.tile = r / size;
  w.head = g * per_group + r % size;
  return w;
}

// n: number of steps of the longest block. uniform: every block has the same work (no mask), so one head at a time.
// all: windowed masks, whose global tiles outlast the others by far more than the rule assumes.
inline int heads_per_group(int n, int n_heads, bool uniform, bool all) {
  if (all) return n_heads;
  const int m = uniform ? 1 : (296 + n) / (n + 1);
  const int groups = n_heads / m > 0 ? n_heads / m : 1;
  return (n_heads + groups - 1) / groups;
}

}  // namespace zx
