// The order in which the decode step kernel asks for the boxes of its ring, as plain functions of numbers: the kernel and a
// model of the ring that runs on the host share them.
//
// Position p of an op's sequence uses stage p % stages, and everybody waits by phase parity, which cannot tell a phase from
// the one two before it.  A consumer that waits for position p is right only if the stage's use two before, p - 2 stages,
// has been released.  What it knows is that its own position before, i, has been filled, hence asked for; so that must imply
// that p - stages may be asked for, too.  Position i therefore waits for all positions up to i - distance, with i - distance
// >= p - stages wherever a consumer goes from i to p.
#pragma once

#ifdef __CUDACC__
#define MLD_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define MLD_HOST_DEVICE inline
#endif

namespace mld {

// Projections: a warp goes from position i to i + warps.
MLD_HOST_DEVICE int ring_distance(int stages, int warps) { return stages - warps; }

// Attention: a warp's items are pairs of positions, 2 warps apart: from the later one of a pair to the earlier one of the next
// (2 warps - 1 on; no further than the ring is long with shorter ones, where the earlier position was this warp's own),
// then to the position behind it.
MLD_HOST_DEVICE int ring_attn_warps(int stages, int warps) { return stages >= 2 * warps - 1 ? warps : stages / 2; }
MLD_HOST_DEVICE int ring_attn_distance(int stages, int attn_warps) {
  return stages >= 2 * attn_warps ? stages - 2 * attn_warps + 1 : stages - 1;
}

// Lanes whose positions lane's own waits for; it may ask when none of them is waiting for its stage.  (A lane per position,
// `stages` of them in a pass; all positions of earlier passes have been asked for.)
MLD_HOST_DEVICE unsigned ring_lanes_before(int lane, int distance) {
  return lane < distance ? 0u : (2u << (lane - distance)) - 1u;
}

}  // namespace mld
