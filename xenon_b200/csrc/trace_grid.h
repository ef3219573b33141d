// trace_grid.h — how a bounce's ray queue is divided over the launch that traces it. Plain C++ as
// well, for the CPU test of the rule.
#pragma once

#if defined(__CUDACC__)
#define XB_GRID_HD __host__ __device__ __forceinline__
#else
#define XB_GRID_HD inline
#endif

namespace xb {

// A traversal launch: its blocks of four warps, and the warps a short queue is spread over, which
// are those of the launch that fit on the GPU at once. With all that fit on the GPU instead, a launch
// of fewer left lanes idle for its whole time while rays waited (B200, 1080p, one mesh of 1.31 M
// triangles, 4 of 8 shadow blocks an SM: 1.407 -> 1.396 ms per sample; 261 instances, 4 blocks an SM
// for both kinds of ray: 4.786 -> 4.749; others within 0.2 %).
struct TraceGrid {
  int blocks, warps;
};
// tuned: the blocks the tuning asks for; occ: the blocks of the launched kernel that fit on an SM;
// per_thread: one ray per thread, whose blocks beyond the resident ones queue.
XB_GRID_HD TraceGrid trace_grid(int tuned, int num_sms, int occ, bool per_thread) {
  const int fit = num_sms * occ < tuned ? num_sms * occ : tuned;
  TraceGrid g;
  g.blocks = per_thread ? tuned : fit;
  g.warps = 4 * fit;
  return g;
}

// The lanes of each warp that take rays from a queue of n.
XB_GRID_HD int queue_lanes(int n, int warps) {
  const int k = (n + warps - 1) / warps;
  return k < 1 ? 1 : (k > 32 ? 32 : k);
}

}  // namespace xb
