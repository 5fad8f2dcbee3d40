// Decode-stage dequant-GEMV, streaming form (1..32 tokens per launch) over the
// reference's packed weight layout [K/4][N/4][4 k][4 n].
//
// The kernel is HBM-bound, so it is organised around keeping the memory system
// busy and the exit path short:
//  * the grid is one CTA per SM (two for matrices of several passes); each CTA
//    owns a strip of output columns (16-byte granularity, so the strips balance
//    to within one chunk) and streams every K row of that strip - no split-K
//    traffic through global memory.  When the matrix is too narrow for 148 useful strips, the CTAs of
//    a thread-block cluster (two, or up to eight for one token) share a strip, take an even part of K each
//    and combine through distributed shared memory;
//  * packed weights (128-byte-swizzled boxes), block scales and activations are
//    staged by TMA / bulk copies into a ring of shared-memory stages, all
//    completing on one mbarrier per stage;
//  * eight consumer warps dequantise in registers and feed m16n8k16 tensor-core
//    MMAs (weights as the 16-row operand, tokens as columns), fp32 accumulate;
//    a single token goes through integer MMAs on 16-bit fixed-point activations
//    instead (the DIGITS form below);
//  * with programmatic dependent launch the next GEMV starts streaming its
//    weights while this one drains; only the activation loads wait for the
//    predecessor.
//
// Arithmetic restated from GetFullyConnectedKernelCode
// (ml_drift/common/kernels/fully_connected.cc:623-942) and fc:: helpers
// (fully_connected_util.cc:80-229, 356-407); accumulation is fp32 for both
// fp16 precision modes.
#include <cuda_fp16.h>

#include <cstdlib>

#include "common.cuh"
#include "kernels.h"

namespace mld {

namespace {

constexpr int kConsumerWarps = 8;
constexpr int kStageRows = kConsumerWarps * 8;  // k-slices per stage (256 input channels)
constexpr int kBoxBytes = kStageRows * 128;     // one weight box: 64 rows x 128 bytes

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same from other accumulators: d = a b + c.
__device__ __forceinline__ void mma_f16_from(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ void mma_u8s8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t lop3_and_or(uint32_t x, uint32_t mask, uint32_t orv) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(r) : "r"(x), "r"(mask), "r"(orv));  // (x & mask) | orv
  return r;
}
__device__ __forceinline__ uint32_t hsub2_u32(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

// Fragment geometry.  Lane = 4*g + t.  One warp step covers four k-slice rows
// (row of lane = base + 2*t + parity) of one 128-byte box row; lane g owns 16
// bytes (one "chunk") of it.
//   BITS 4: a chunk = two 4x4 blocks (8 outputs) -> 4 MMAs, 64 outputs per box
//   BITS 8: a chunk = one 4x4 block  (4 outputs) -> 2 MMAs, 32 outputs per box
// MMA f of a lane: rows g / g+8 are outputs NPL*g + 2*f + {0,1} of the box; the
// sixteen k columns are (row t: k0 k1) at 2t,2t+1 and (row t: k2 k3) at 2t+8,9.
template <int BITS>
struct Frag {
  static constexpr int NF = BITS == 4 ? 4 : 2;   // MMAs (accumulator fragments) per lane and box
  static constexpr int NPL = BITS == 4 ? 8 : 4;  // outputs per chunk
  static constexpr int BOX_N = NPL * 8;          // outputs per box (64 / 32)
};

// EXACT operands: (1024 + u) with the offset removed by one packed half
// subtract, giving the signed weight exactly (x16 for high nibbles).
// SUBNORMAL operands: the raw masked bits, i.e. fp16 subnormals u * 2^-24 (x16
// for high nibbles); the "- shift * sum(x)" term comes from one extra MMA per
// step against a constant operand, whose result the products are then added to,
// and results carry a 2^-24 factor.
// The A operand of MMA f from a lane's 16 bytes (f is a constant wherever this is inlined).
template <int BITS, bool SUBNORMAL>
__device__ __forceinline__ void unpack(const uint4& q, int f, uint32_t (&a)[4]) {
  if constexpr (BITS == 4) {
    // blockA.lo(k0k1) blockA.hi(k2k3) blockB.lo blockB.hi
    const uint32_t lo = f < 2 ? q.x : q.z, hi = f < 2 ? q.y : q.w;
    const uint32_t l = (f & 1) ? lo >> 8 : lo, h = (f & 1) ? hi >> 8 : hi;
    if constexpr (SUBNORMAL) {
      a[0] = l & 0x000F000Fu;
      a[1] = l & 0x00F000F0u;
      a[2] = h & 0x000F000Fu;
      a[3] = h & 0x00F000F0u;
    } else {
      const uint32_t kLo = 0x64086408u;  // half2(1032): 1024 + 8
      const uint32_t kHi = 0x64806480u;  // half2(1152): 1024 + 16*8
      a[0] = hsub2_u32(lop3_and_or(l, 0x000F000Fu, 0x64006400u), kLo);
      a[1] = hsub2_u32(lop3_and_or(l, 0x00F000F0u, 0x64006400u), kHi);
      a[2] = hsub2_u32(lop3_and_or(h, 0x000F000Fu, 0x64006400u), kLo);
      a[3] = hsub2_u32(lop3_and_or(h, 0x00F000F0u, 0x64006400u), kHi);
    }
  } else {
    // bytes: q.x = k0:(n0..n3), q.y = k1, q.z = k2, q.w = k3
    const uint32_t sel = f == 0 ? 0x5140u : 0x7362u;   // outputs 0, 1 or 2, 3
    const uint32_t k01 = prmt(q.x, q.y, sel), k23 = prmt(q.z, q.w, sel);  // [k0 n, k1 n, k0 n+1, k1 n+1], ...
    if constexpr (SUBNORMAL) {
      a[0] = prmt(k01, 0u, 0x4140u);
      a[1] = prmt(k01, 0u, 0x4342u);
      a[2] = prmt(k23, 0u, 0x4140u);
      a[3] = prmt(k23, 0u, 0x4342u);
    } else {
      const uint32_t kM = 0x64646464u;
      const uint32_t kOff = 0x64806480u;  // half2(1152) = 1024 + 128
      a[0] = hsub2_u32(prmt(k01, kM, 0x4140u), kOff);
      a[1] = hsub2_u32(prmt(k01, kM, 0x4342u), kOff);
      a[2] = hsub2_u32(prmt(k23, kM, 0x4140u), kOff);
      a[3] = hsub2_u32(prmt(k23, kM, 0x4342u), kOff);
    }
  }
}

// The bytes of a 4x4 block turned round: word i of `out` is byte i of the four words.
__device__ __forceinline__ void transpose_bytes(const uint4& q, uint32_t (&out)[4]) {
  const uint32_t a = prmt(q.x, q.y, 0x5140u), b = prmt(q.x, q.y, 0x7362u);
  const uint32_t c = prmt(q.z, q.w, 0x5140u), d = prmt(q.z, q.w, 0x7362u);
  out[0] = prmt(a, c, 0x5410u);
  out[1] = prmt(a, c, 0x7632u);
  out[2] = prmt(b, d, 0x5410u);
  out[3] = prmt(b, d, 0x7632u);
}

// --------------------------------------------------------- cluster primitives
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 128; ++i)
      if (mbar_try_wait_cluster(bar, parity)) return true;
    if (globaltimer_ns() - t0 > kWaitLimitNs) return false;
  }
}

#define MLD_CONSUMER_BARRIER() asm volatile("bar.sync 1, %0;" ::"n"(kConsumerWarps * 32) : "memory")

// W: weight boxes per stage (strip width up to W * 128 bytes per pass).
// MONE: single-token launch (only token column 0 is kept).
// DIGITS (one token): integer MMAs instead.  The whole activation vector is fetched once, and before the first stage is
// consumed the warps turn every unit of 32 inputs into fixed point with a power-of-two scale of its own, in signed 8-bit
// digits.  One m16n8k32 u8 x s8 MMA per 16 outputs and unit then multiplies the stored weights (4 bits: as the bytes of the
// reference layout, which hold two outputs each; 8 bits: bytes of a block turned round) by the unit's digits, a B column
// each, so that four (two) units share accumulators.  A 4-bit stage costs 64 MMAs where the fp16 form needs 144, an 8-bit
// stage 32 against 96, and an fp16 MMA occupies the pipe twice as long.  Products and sums of a unit are exact in int32.
//  * 4-bit weights: 16-bit fixed point, x ~ s (256 hi + lo), an input's error at most 2^-15 of the unit's largest.
//  * 8-bit weights: 32-bit fixed point in four digits, an input's error at most 2^-31 of the unit's largest, which is below
//    what the fp32 sums of the fp16 form lose (its terms are up to 255 x, their offset 128 x taken off at the end).  2048
//    inputs, one in 32 of them 300 with zero weights: error against 64 bits 2.1e-4, the rounding of the output; two digits
//    4.5e-3, the fp16 form 2.2e-4.  151936 x 2048 in a graph: 49.1 us; two digits 47.3, the fp16 form 55.8.
// SPLIT: more than eight tokens (an MMA's columns) are split over the warps: 2^ts_shift warps share 8 << ts_shift k-slice rows
// of a stage and take eight tokens each.  They unpack the same weights, which costs less than the MMAs, and a lane's
// accumulators stay eight tokens wide, so that two CTAs still fit an SM.
// ZP: a zero point per scale; a second box of the scales' shape follows them in the stage.  (u - 8 - z) s x summed
// over a group is s (sum(u x) - (1 + z / 8) 8 sum(x)), so the zero point only scales the offset term, in fp32
// (2048 x 4096 INT4, 12 tokens: 10.3 us; the general kernel, which took such weights before, 45.8).  One token stays in the
// fp16 form: these launches wait before they read anything, so the digits have no stream to hide behind (2048 x 4096 in a
// graph 6.0 us, two digits 6.2, four 6.5).
// INTERLEAVE: the passes of all strips lie side by side (StripGeometry::interleave).  A form of its own, because the steps
// and box counts that only it has, worked out at run time, cost every other launch 0.3 to 0.8 us (14208 x 2432 INT4, one
// token 13.6 against 12.9; 4096 x 11008 10.9 against 10.2).  Several tokens through strips of two boxes take this form always:
// they have nothing to interleave, but the compiler's schedule of it is the faster one (4096 x 11008, 5 tokens: 15.0 against
// 15.4).
// CUT: clusters of more than two CTAs cut K (StripGeometry::ksplit).  A form of its own likewise: adding up any number of
// partners' sums cost launches of one or two CTAs to a strip 0.1 to 0.3 us (896 x 12288 4.15 / 4.35, 2432 x 6048 INT8 6.05 /
// 6.47).
template <int BITS, int W, bool SUBNORMAL, bool MONE, bool DIGITS, bool ZP, bool SPLIT, bool INTERLEAVE, bool CUT>
__global__ void __launch_bounds__((kConsumerWarps + 1) * 32, W <= 2 ? 2 : 1)
    fc_strip_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_s,
                    const __grid_constant__ CUtensorMap tmap_z, StripArgs a) {
  using F = Frag<BITS>;
  static_assert(!ZP || SUBNORMAL, "the offset term comes from the constant operand of the subnormal form");
  constexpr int WT = W * F::BOX_N;       // outputs per pass
  constexpr int NJ = MONE ? 2 : 4;       // accumulator values kept per fragment
  constexpr int ND = BITS == 4 ? 2 : 4;  // DIGITS: digits of an activation
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* red = reinterpret_cast<float*>(smem + (size_t)a.stages * a.stage_bytes);  // [warps][WT][red_m]
  float* peer = red + kConsumerWarps * WT * a.red_m;                                // [partners][WT][peer_m]
  const int partners = CUT ? a.ksplit - 1 : 1;
  uint64_t* full = reinterpret_cast<uint64_t*>(peer + ((partners * WT * a.peer_m + 1) & ~1));
  uint64_t* empty = full + a.stages;
  uint64_t* peer_bar = empty + a.stages;
  // DIGITS: the activation vector of this CTA's K range as digits ([unit][digit, the highest first][8 words], word j = the
  // four inputs of k-slice j), the vector itself (two digits take its place), then per unit and pair of digits {bits of
  // the pair's scale, its offset: 8 (128) x the sum of the pair's integers}
  uint64_t* xbar = peer_bar + 1;
  uint8_t* xdig = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(xbar + 1) + 15) & ~uintptr_t(15));
  uint8_t* xraw = ND == 4 ? xdig + (size_t)a.rows_per_split * 16 : xdig;
  uint2* xmeta = reinterpret_cast<uint2*>(xraw + (size_t)a.rows_per_split * 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kr = a.ksplit > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int strip = blockIdx.x / a.ksplit;

  // strip -> chunk range (16-byte chunks of a weight row), balanced to one unit
  const int64_t u_lo = (int64_t)strip * a.units / a.strips, u_hi = (int64_t)(strip + 1) * a.units / a.strips;
  // (interleaved: the passes of all strips side by side, pass p of strip s being the grid's (p strips + s)-th box or
  // pair of boxes, so that what the SMs read at a time is one contiguous piece of every weight row)
  const bool interleave = INTERLEAVE && a.interleave;
  const int cs = interleave ? strip * W * 8 : static_cast<int>(u_lo) * a.gran;
  const int ce = interleave ? a.units * a.gran : static_cast<int>(u_hi) * a.gran;
  const int pass_step = interleave ? a.strips * W * 8 : W * 8;
  const int passes = (ce - cs + pass_step - 1) / pass_step;
  const int r_lo = kr * a.rows_per_split;
  const int r_hi = min(a.src_slices, r_lo + a.rows_per_split);
  const int n_st = (r_hi - r_lo + kStageRows - 1) / kStageRows;

#ifdef MLD_TRACE  // per-CTA timestamps for tuning, compiled in only on request
  unsigned long long* tr = a.trace != nullptr ? a.trace + (size_t)blockIdx.x * 8 : nullptr;
#else
  constexpr unsigned long long* tr = nullptr;
#endif
  // The producer thread initialises the barriers and goes straight on to issue
  // its first loads; the consumers wait for the initialisation on a named
  // barrier the producer warp only arrives at.
  if (warp == kConsumerWarps) {
    if (lane == 0) {
      if (tr) tr[0] = globaltimer_ns();
      for (int s = 0; s < a.stages; ++s) {
        mbar_init(&full[s], 1);
        mbar_init(&empty[s], kConsumerWarps);
      }
      mbar_init(peer_bar, partners * kConsumerWarps * 32);
      if constexpr (DIGITS) mbar_init(xbar, 1);
      fence_barrier_init();
    }
    __syncwarp();
    asm volatile("bar.arrive 2, %0;" ::"n"((kConsumerWarps + 1) * 32) : "memory");
  } else {
    asm volatile("bar.sync 2, %0;" ::"n"((kConsumerWarps + 1) * 32) : "memory");
  }
  // cluster partners: arrive now, wait only before the first remote access
  if (a.ksplit > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  if (a.pdl == kPdlOverlap || a.pdl == kPdlIndependent) pdl_launch_dependents();

  if (warp == kConsumerWarps) {
    // ------------------------------------------------------------ producer
    if (n_st > 0) {
      const uint64_t pol = policy_evict_first();
      const int total = passes * n_st;
      const uint32_t s_bytes = a.scale_rows > 0 ? static_cast<uint32_t>(a.scale_rows) * WT * (ZP ? 4u : 2u) : 0u;
      auto issue_weights = [&](int item, int stage) {
        const int pass = item / n_st, si = item % n_st;
        uint8_t* st = smem + (size_t)stage * a.stage_bytes;
        const int row0 = r_lo + si * kStageRows;
        const int rows = min(kStageRows, r_hi - row0);
        const int chunk0 = cs + pass * pass_step;
        // (boxes past the end of the matrix, in the last pass, are not fetched: their sums, of whatever the stage held, are
        // not stored)
        const int boxes = INTERLEAVE ? min(W, (ce - chunk0 + 7) / 8) : W;
        mbar_arrive_expect_tx(&full[stage], boxes * kBoxBytes + s_bytes +
                                                (DIGITS ? 0u : static_cast<uint32_t>(rows) * a.M_total * 8u));
#pragma unroll
        for (int b = 0; b < W; ++b)
          if (b < boxes) tma_load_2d_hint(st + b * kBoxBytes, &tmap_w, &full[stage], (chunk0 + b * 8) * 16, row0, pol);
        if (a.scale_rows > 0) {
          tma_load_2d(st + W * kBoxBytes, &tmap_s, &full[stage], chunk0 * F::NPL, row0 / a.group_slices);
          if constexpr (ZP)
            tma_load_2d(st + W * kBoxBytes + a.zp_off, &tmap_z, &full[stage], chunk0 * F::NPL, row0 / a.group_slices);
        }
      };
      auto issue_x = [&](int item, int stage) {
        if constexpr (DIGITS) return;  // the whole vector is fetched once, below
        const int si = item % n_st;
        uint8_t* st = smem + (size_t)stage * a.stage_bytes;
        const int row0 = r_lo + si * kStageRows;
        const int rows = min(kStageRows, r_hi - row0);
        bulk_load_1d(st + W * kBoxBytes + a.scale_stage_bytes,
                     static_cast<const uint8_t*>(a.x) + (size_t)row0 * a.M_total * 8,
                     static_cast<uint32_t>(rows) * a.M_total * 8u, &full[stage]);
      };
      // weights and scales are constants: the first ring-full of them is
      // requested before waiting for the preceding kernel; activations after.
      // Launches that overlap completely, or not at all, request the whole ring at once, one lane per stage.  A launch that
      // hands over at the activation load requests it stage by stage: measured, its burst only gets in the way
      // of the launch ahead of it, which is still streaming.
      const int head = total < a.stages ? total : a.stages;
      if (a.pdl >= kPdlIndependent) {
        if (a.pdl == kPdlWaitFirst) pdl_wait();
        if (lane < head) issue_weights(lane, lane);
        __syncwarp();
      }
      if (lane != 0) return;
      if (a.pdl < kPdlIndependent)
        for (int it = 0; it < head; ++it) issue_weights(it, it);
      if (tr) tr[1] = globaltimer_ns();
      if (a.pdl == kPdlOverlap) pdl_wait();  // (independent: the caller declared x and y untouched by the launch before)
      if (a.wait.world > 1) {
        const unsigned seq = static_cast<unsigned>(*a.wait.step * a.wait.seq_per_step + a.wait.seq_off);
        if (!wait_peer_flags(a.wait.flags, a.wait.world, seq, a.wait.limit_ns)) atomicExch(a.error, kErrPeerWait);
      }
      if (tr) tr[2] = globaltimer_ns();
      if constexpr (DIGITS) {
        const uint32_t xbytes = static_cast<uint32_t>(r_hi - r_lo) * 8u;
        mbar_arrive_expect_tx(xbar, xbytes);
        bulk_load_1d(xraw, static_cast<const uint8_t*>(a.x) + (size_t)r_lo * 8, xbytes, xbar);
      }
      for (int it = 0; it < head; ++it) issue_x(it, it);
      int stage = head == a.stages ? 0 : head;
      uint32_t phase = head == a.stages ? 1 : 0;
      for (int it = head; it < total; ++it) {
        if (!mbar_wait(&empty[stage], phase ^ 1)) {
          atomicExch(a.error, 1);
          break;
        }
        issue_weights(it, stage);
        issue_x(it, stage);
        if (++stage == a.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      // Everything this CTA needs has been requested: use the memory system's
      // idle tail (epilogue, the glue kernels that follow) to pull this CTA's
      // share of the next projection's weights into L2.
      // Launches that did not wait above still complete in stream order: the grid is not done before the
      // grid ahead of it is.
      if (a.pdl == kPdlIndependent) pdl_wait();
      if (a.next_w != nullptr) {
        const unsigned long long per = ((a.next_w_bytes / gridDim.x) + 127ull) & ~127ull;
        unsigned long long lo = per * blockIdx.x, hi = lo + per;
        if (hi > a.next_w_bytes) hi = a.next_w_bytes & ~15ull;
        for (; lo < hi; lo += 16384ull) {
          const unsigned long long n = hi - lo < 16384ull ? hi - lo : 16384ull;
          bulk_prefetch_l2(static_cast<const uint8_t*>(a.next_w) + lo, static_cast<uint32_t>(n & ~15ull));
        }
      }
    }
    return;
  }

  // -------------------------------------------------------------- consumers
  const int g = lane >> 2, t = lane & 3;
  // minus the offset as a subnormal: -8 / -128 against rows g; rows g + 8 (high nibbles) carry it x16
  constexpr uint32_t kOffsetA = BITS == 4 ? 0x80088008u : 0x80808080u, kOffsetA16 = 0x80808080u;
  constexpr float kOdd = BITS == 4 ? 0.0625f : 1.0f;                  // high nibbles are carried x16
  constexpr float kOutScale = (SUBNORMAL && !DIGITS) ? 16777216.0f : 1.0f;
  int stage = 0;
  uint32_t phase = 0;
  bool failed = false;
#ifdef MLD_TRACE
  long long tr_wait_cycles = 0, tr_busy_cycles = 0;
#endif

  if constexpr (DIGITS) {
    if (n_st > 0) {
      if (!mbar_wait(xbar, 0)) {
        atomicExch(a.error, 2);
        failed = true;
      }
      // this warp digitises unit si * 8 + warp of every stage si; lane = 4 * (stage of the round) + chunk, a chunk
      // being eight inputs (k-slices 2q and 2q + 1 of the unit)
      for (int si0 = 0; si0 < n_st && !failed; si0 += 8) {
        const int si = si0 + (lane >> 2), q = lane & 3;
        const bool have = si < n_st;
        const int u = si * 8 + warp;
        const int row = r_lo + u * 8 + 2 * q;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (have && row < r_hi) {
          v = *reinterpret_cast<const uint4*>(xraw + (size_t)u * 64 + q * 16);
          if (row + 1 >= r_hi) v.z = v.w = 0u;
        }
        __syncwarp();  // the unit's four lanes have read before any of them rewrites it
        float xf[8];
        {
          const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
          const float2 f1 = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
          const float2 f2 = __half22float2(*reinterpret_cast<const __half2*>(&v.z));
          const float2 f3 = __half22float2(*reinterpret_cast<const __half2*>(&v.w));
          xf[0] = f0.x; xf[1] = f0.y; xf[2] = f1.x; xf[3] = f1.y;
          xf[4] = f2.x; xf[5] = f2.y; xf[6] = f3.x; xf[7] = f3.y;
        }
        float amax = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(xf[i]));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        // the smallest power of two s with amax / s <= 32512 (a float with an empty mantissa); 1 / s is exact
        uint32_t sbits = (__float_as_uint(amax * (1.0f / 32512.0f)) + 0x007FFFFFu) & 0x7F800000u;
        if (sbits < (16u << 23)) sbits = 16u << 23;
        const float inv = __uint_as_float((254u << 23) - sbits);
        // an infinity or NaN among the unit's inputs (an all-ones fp16 exponent) has no digits: the unit's scale
        // becomes NaN, and with it every output, as the reference arithmetic would make most of them
        const auto non_finite = [](uint32_t w) { return (w & 0x7C00u) == 0x7C00u || (w & 0x7C000000u) == 0x7C000000u; };
        unsigned bad = (non_finite(v.x) || non_finite(v.y) || non_finite(v.z) || non_finite(v.w)) ? 1u : 0u;
        bad |= __shfl_xor_sync(0xffffffffu, bad, 1);
        bad |= __shfl_xor_sync(0xffffffffu, bad, 2);
        if constexpr (ND == 4) {
          // x 65536 / s rounded (|.| <= 127 x 2^24), plus 2^7, 2^15 and 2^23: its bytes are the digits, the lower three ^ 0x80
          uint32_t w[2][4];  // [k-slice][byte]: the four inputs of that byte
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            uint32_t z[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) z[i] = static_cast<uint32_t>(__float2int_rn(xf[4 * e + i] * inv * 65536.0f)) + 0x00808080u;
            transpose_bytes(make_uint4(z[0], z[1], z[2], z[3]), w[e]);
#pragma unroll
            for (int b = 0; b < 3; ++b) w[e][b] ^= 0x80808080u;
          }
          int isum[2];  // of the high pair of digits and of the low one
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int b = 3 - 2 * h;
            int v2 = __dp4a(static_cast<int>(w[0][b]), 0x01010101, 0);
            v2 = __dp4a(static_cast<int>(w[1][b]), 0x01010101, v2) * 256;
            v2 = __dp4a(static_cast<int>(w[0][b - 1]), 0x01010101, v2);
            v2 = __dp4a(static_cast<int>(w[1][b - 1]), 0x01010101, v2);
            v2 += __shfl_xor_sync(0xffffffffu, v2, 1);
            isum[h] = v2 + __shfl_xor_sync(0xffffffffu, v2, 2);
          }
          if (have) {
            uint32_t* ud = reinterpret_cast<uint32_t*>(xdig + (size_t)u * 128);
#pragma unroll
            for (int b = 0; b < 4; ++b) *reinterpret_cast<uint2*>(ud + (3 - b) * 8 + 2 * q) = make_uint2(w[0][b], w[1][b]);
            if (q == 0) {
              xmeta[2 * u] = make_uint2(bad ? 0x7FC00000u : sbits, static_cast<uint32_t>(128 * isum[0]));
              xmeta[2 * u + 1] = make_uint2(sbits - (16u << 23), static_cast<uint32_t>(128 * isum[1]));  // (bytes = weights + 128)
            }
          }
        } else {
          // z = round(x / s) + 128 in the low 16 bits of the sum's mantissa: byte 1 = high digit, byte 0 ^ 0x80 = low digit
          uint32_t z[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) z[i] = __float_as_uint(fmaf(xf[i], inv, 12583040.0f));
          uint32_t hiw[2], low[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const uint32_t h01 = prmt(z[4 * e], z[4 * e + 1], 0x0051u), h23 = prmt(z[4 * e + 2], z[4 * e + 3], 0x0051u);
            const uint32_t l01 = prmt(z[4 * e], z[4 * e + 1], 0x0040u), l23 = prmt(z[4 * e + 2], z[4 * e + 3], 0x0040u);
            hiw[e] = prmt(h01, h23, 0x5410u);
            low[e] = prmt(l01, l23, 0x5410u) ^ 0x80808080u;
          }
          int isum = __dp4a(static_cast<int>(hiw[0]), 0x01010101, 0);
          isum = __dp4a(static_cast<int>(hiw[1]), 0x01010101, isum) * 256;
          isum = __dp4a(static_cast<int>(low[0]), 0x01010101, isum);
          isum = __dp4a(static_cast<int>(low[1]), 0x01010101, isum);
          isum += __shfl_xor_sync(0xffffffffu, isum, 1);
          isum += __shfl_xor_sync(0xffffffffu, isum, 2);
          if (have) {
            uint32_t* ud = reinterpret_cast<uint32_t*>(xdig + (size_t)u * 64);
            *reinterpret_cast<uint2*>(ud + 2 * q) = make_uint2(hiw[0], hiw[1]);
            *reinterpret_cast<uint2*>(ud + 8 + 2 * q) = make_uint2(low[0], low[1]);
            if (q == 0) xmeta[u] = make_uint2(bad ? 0x7FC00000u : sbits, static_cast<uint32_t>(8 * isum));  // (nibbles = weights + 8)
          }
        }
      }
    }
    MLD_CONSUMER_BARRIER();  // a warp multiplies by units other warps digitised
  }

  for (int pass = 0; pass < passes && !failed; ++pass) {
    float tot[W][F::NF][NJ];
#pragma unroll
    for (int b = 0; b < W; ++b)
#pragma unroll
      for (int f = 0; f < F::NF; ++f)
#pragma unroll
        for (int j = 0; j < NJ; ++j) tot[b][f][j] = 0.0f;
    [[maybe_unused]] const int boxes = INTERLEAVE ? min(W, (ce - cs - pass * pass_step + 7) / 8) : W;  // of this pass

    for (int si = 0; si < n_st; ++si) {
#ifdef MLD_TRACE
      const long long tw0 = clock64();
#endif
      if (!mbar_wait(&full[stage], phase)) {
        atomicExch(a.error, 2);
        failed = true;
        break;
      }
#ifdef MLD_TRACE
      const long long tw1 = clock64();
      tr_wait_cycles += tw1 - tw0;
      if (a.trace_skip_math) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[stage]);
        if (++stage == a.stages) {
          stage = 0;
          phase ^= 1;
        }
        continue;
      }
#endif
      if (tr && threadIdx.x == 0 && pass == 0 && si == 0) tr[3] = globaltimer_ns();
      const uint8_t* st = smem + (size_t)stage * a.stage_bytes;
      const uint8_t* xs = st + W * kBoxBytes + a.scale_stage_bytes;
      const int row0 = r_lo + si * kStageRows;
      if constexpr (DIGITS) {
        static_assert(MONE && !ZP, "the digit form is for one token and weights without zero points");
        // A stage is 2 W tasks: (half of its 64 k-slice rows = four units) x (box of 64 outputs).  The four
        // units of a task share accumulators: B column 2 j holds the high and 2 j + 1 the low digits of unit j
        // (lanes g supply column g, zero for the other units), so after the units' MMAs lane t holds both
        // digit sums of unit t and finishes that unit.  With fewer tasks than warps, groups of warps take
        // the stages in turn; every warp still waits for and releases every stage.
        constexpr int T = W == 3 ? 8 : 2 * W;
        constexpr int GC = kConsumerWarps / T;
        const int task = warp % T, tb = task >> 1, hq = task & 1;
        if (tb < boxes && si % GC == warp / T) {
          const int ubase = si * 8 + hq * 4;  // the task's first unit within the CTA's K range
          constexpr int U = 8 / ND;  // units that share a set of accumulators
          uint32_t bm[4 / U][2];
          int accs[4 / U][F::NF][4];
#pragma unroll
          for (int p = 0; p < 4 / U; ++p) {
            const uint32_t* ud = reinterpret_cast<const uint32_t*>(xdig) + ((size_t)(ubase + p * U + g / ND) * ND + g % ND) * 8;
            bm[p][0] = ud[t];
            bm[p][1] = ud[4 + t];
#pragma unroll
            for (int f = 0; f < F::NF; ++f) accs[p][f][0] = accs[p][f][1] = accs[p][f][2] = accs[p][f][3] = 0;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            // k-slice rows ra and ra + 4 of unit j are what lane t feeds the MMA's K with
            const int ra = 32 * hq + 8 * j + t, rb = ra + 4;
            const uint4 qa = *reinterpret_cast<const uint4*>(st + tb * kBoxBytes + ra * 128 + ((g ^ (ra & 7)) << 4));
            const uint4 qb = *reinterpret_cast<const uint4*>(st + tb * kBoxBytes + rb * 128 + ((g ^ (rb & 7)) << 4));
            const bool mine = g / ND == j % U;
            const uint32_t b0 = mine ? bm[j / U][0] : 0u, b1 = mine ? bm[j / U][1] : 0u;
            int(&acc)[F::NF][4] = accs[j / U];
            if constexpr (BITS == 4) {
#pragma unroll
              for (int f = 0; f < 4; ++f) {
                // outputs 2f (low nibbles) and 2f + 1 (high nibbles) of this lane's eight: byte i of a block word is
                // input i / 2, output pair i % 2, so the four inputs of a pair are bytes 0, 2 (or 1, 3) of the two words
                const uint32_t sel = (f & 1) ? 0x7531u : 0x6420u;
                const uint32_t wa = f < 2 ? prmt(qa.x, qa.y, sel) : prmt(qa.z, qa.w, sel);
                const uint32_t wb = f < 2 ? prmt(qb.x, qb.y, sel) : prmt(qb.z, qb.w, sel);
                // rows g take the whole byte (even output + 16 x odd output), rows g + 8 the odd output x 16
                const uint32_t af[4] = {wa, wa & 0xF0F0F0F0u, wb, wb & 0xF0F0F0F0u};
                mma_u8s8(acc[f], af, b0, b1);
              }
            } else {
              // a block is four inputs (words) x four outputs (bytes): turned round, a word is an output's four inputs
              uint32_t wa[4], wb[4];
              transpose_bytes(qa, wa);
              transpose_bytes(qb, wb);
#pragma unroll
              for (int f = 0; f < 2; ++f) {
                const uint32_t af[4] = {wa[2 * f], wa[2 * f + 1], wb[2 * f], wb[2 * f + 1]};  // rows g, g + 8: outputs 2f, 2f + 1
                mma_u8s8(acc[f], af, b0, b1);
              }
            }
          }
          // lane t finishes columns 2t and 2t + 1, a pair of digits of one unit: the pair's scale and offset, the weight
          // scales of the unit's group
#pragma unroll
          for (int p = 0; p < 4 / U; ++p) {
            const int unit = p * U + 2 * t / ND, pair = t % (ND / 2);  // of the task's four
            const int(&acc)[F::NF][4] = accs[p];
            const uint2 meta = xmeta[(ubase + unit) * (ND / 2) + pair];
            const float sx = __uint_as_float(meta.x);
            const int off = static_cast<int>(meta.y);
            float sc[F::NPL];
            const int gidx = a.gs_shift >= 0 ? ((32 * hq + 8 * unit) >> a.gs_shift) : 0;
            if (a.scale_rows > 0) {
              const __half* sp = reinterpret_cast<const __half*>(st + W * kBoxBytes) + gidx * WT + tb * F::BOX_N + F::NPL * g;
#pragma unroll
              for (int i = 0; i < F::NPL / 4; ++i) {
                const uint2 w = reinterpret_cast<const uint2*>(sp)[i];
                const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&w.x));
                const float2 f1 = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
                sc[4 * i] = f0.x; sc[4 * i + 1] = f0.y; sc[4 * i + 2] = f1.x; sc[4 * i + 3] = f1.y;
              }
            } else {
#pragma unroll
              for (int i = 0; i < F::NPL; ++i) sc[i] = a.scalar_scale;
            }
            // acc: {row g high digit, row g low, row g + 8 high, row g + 8 low} of the pair
#pragma unroll
            for (int f = 0; f < F::NF; ++f) {
              int even, odd;
              if constexpr (BITS == 4) {
                even = (acc[f][0] - acc[f][2]) * 256 + (acc[f][1] - acc[f][3]) - off;
                odd = ((acc[f][2] * 256 + acc[f][3]) >> 4) - off;
              } else {  // (|sum| <= 32 * 255 * 32640 < 2^28)
                even = acc[f][0] * 256 + acc[f][1] - off;
                odd = acc[f][2] * 256 + acc[f][3] - off;
              }
              tot[0][f][0] = fmaf(sc[2 * f] * sx, static_cast<float>(even), tot[0][f][0]);
              tot[0][f][1] = fmaf(sc[2 * f + 1] * sx, static_cast<float>(odd), tot[0][f][1]);
            }
          }
        }
      } else {
        // eight rows (two steps) of the stage at a time: one per stage, or the 2^ts_shift of this warp's group
        const int n_rr = SPLIT ? 1 << a.ts_shift : 1, token = (warp & (n_rr - 1)) * 8 + g;
        for (int rr = 0; rr < n_rr; ++rr) {
        const int rbase = ((warp & ~(n_rr - 1)) + rr) * 8;
        uint32_t bx[2][2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const int r = rbase + 2 * t + p;
          bx[p][0] = bx[p][1] = 0u;
          if (row0 + r < r_hi && token < a.M) {
            const uint2 xv = *reinterpret_cast<const uint2*>(xs + ((size_t)r * a.M_total + a.tok0 + token) * 8);
            bx[p][0] = xv.x;
            bx[p][1] = xv.y;
          }
        }
        // minus the offset times the sum of the inputs, x16 for the rows of high nibbles: what the products are added to
        // (zero points: what is added to them, times a factor of each output's own)
        float zero[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        float offset[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if constexpr (SUBNORMAL) {
          const uint32_t oa[4] = {kOffsetA, kOffsetA16, kOffsetA, kOffsetA16};
          mma_f16_from(offset, oa, bx[0][0], bx[0][1], zero);
          mma_f16(offset, oa, bx[1][0], bx[1][1]);
        }
        const int gidx = a.gs_shift >= 0 ? (rbase >> a.gs_shift) : 0;
#pragma unroll
        for (int b = 0; b < W; ++b) {
          float grp[F::NF][4];
#pragma unroll
          for (int p = 0; p < 2; ++p) {
            const int r = rbase + 2 * t + p;
            const uint4 q = *reinterpret_cast<const uint4*>(st + b * kBoxBytes + r * 128 + ((g ^ (r & 7)) << 4));
#pragma unroll
            for (int f = 0; f < F::NF; ++f) {
              uint32_t av[4];
              unpack<BITS, SUBNORMAL>(q, f, av);
              if (p == 0)
                mma_f16_from(grp[f], av, bx[p][0], bx[p][1], ZP ? zero : offset);
              else
                mma_f16(grp[f], av, bx[p][0], bx[p][1]);
            }
          }
          // scales (and zero points) of this lane's outputs for the group these eight rows are in
          float sc[F::NPL], zf[F::NPL];
          const auto load_params = [&](const uint8_t* box, float (&v)[F::NPL]) {
            const __half* sp = reinterpret_cast<const __half*>(box) + gidx * WT + b * F::BOX_N + F::NPL * g;
            uint32_t w[F::NPL / 2];
            if constexpr (BITS == 4) {
              const uint4 sv = *reinterpret_cast<const uint4*>(sp);
              w[0] = sv.x; w[1] = sv.y; w[2] = sv.z; w[3] = sv.w;
            } else {
              const uint2 sv = *reinterpret_cast<const uint2*>(sp);
              w[0] = sv.x; w[1] = sv.y;
            }
#pragma unroll
            for (int i = 0; i < F::NPL / 2; ++i) {
              const float2 f2 = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
              v[2 * i] = f2.x;
              v[2 * i + 1] = f2.y;
            }
          };
          if (a.scale_rows > 0) {
            load_params(st + W * kBoxBytes, sc);
          } else {
#pragma unroll
            for (int i = 0; i < F::NPL; ++i) sc[i] = a.scalar_scale;
          }
          if constexpr (ZP) {
            load_params(st + W * kBoxBytes + a.zp_off, zf);
#pragma unroll
            for (int i = 0; i < F::NPL; ++i) zf[i] = fmaf(zf[i], BITS == 4 ? 0.125f : 0.0078125f, 1.0f);
          }
          if constexpr (BITS == 4) {
#pragma unroll
            for (int f = 0; f < F::NF; ++f) sc[2 * f + 1] *= kOdd;
          }
          // row g of MMA f is output 2f, row g+8 is output 2f+1
#pragma unroll
          for (int f = 0; f < F::NF; ++f) {
#pragma unroll
            for (int jj = 0; jj < NJ; ++jj) {
              const int j = MONE ? 2 * jj : jj;  // MONE keeps (row g, token 2t) and (row g+8, token 2t)
              const int o = 2 * f + (j >> 1);
              float v = grp[f][j];
              if constexpr (ZP) v = fmaf(offset[j], zf[o], v);
              tot[b][f][jj] = fmaf(sc[o], v, tot[b][f][jj]);
            }
          }
        }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage]);
#ifdef MLD_TRACE
      tr_busy_cycles += clock64() - tw1;
#endif
      if (++stage == a.stages) {
        stage = 0;
        phase ^= 1;
      }
    }
    if (failed) break;
#ifdef MLD_TRACE
    if (tr && threadIdx.x == 0) {
      tr[6] = static_cast<unsigned long long>(tr_wait_cycles);
      tr[7] = static_cast<unsigned long long>(tr_busy_cycles);
    }
#endif

    // ------------------------------------------------ pass epilogue
    if (tr && threadIdx.x == 0) tr[4] = globaltimer_ns();
    const int chunk0 = cs + pass * pass_step;
    const int n0 = chunk0 * F::NPL;               // first output of this pass
    const int n_end = min(ce * F::NPL, a.N4);      // one past the last output this CTA owns
    const int n_rr = SPLIT ? 1 << a.ts_shift : 1;
    uint32_t peer_remote = 0, bar_remote = 0;
    if constexpr (DIGITS) {
      // tot[0] is this warp's box (tb) summed over the units the lane finished: add the four lanes t up; the
      // warp contributes nothing to the other boxes
      constexpr int T = W == 3 ? 8 : 2 * W;
      const int tb = (warp % T) >> 1;
#pragma unroll
      for (int f = 0; f < F::NF; ++f)
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
          float v = tot[0][f][jj];
          v += __shfl_xor_sync(0xffffffffu, v, 1);
          v += __shfl_xor_sync(0xffffffffu, v, 2);
          if (t == 0) {
#pragma unroll
            for (int b = 0; b < W; ++b)
              red[(warp * WT + b * F::BOX_N + F::NPL * g + 2 * f + jj) * a.red_m] = b == tb ? v : 0.0f;
          }
        }
    } else {
#pragma unroll
      for (int b = 0; b < W; ++b)
#pragma unroll
        for (int f = 0; f < F::NF; ++f)
#pragma unroll
          for (int jj = 0; jj < NJ; ++jj) {
            const int j = MONE ? 2 * jj : jj;
            const int n_local = b * F::BOX_N + F::NPL * g + 2 * f + ((j >> 1) & 1);
            const int tok = 2 * t + (j & 1);
            if (SPLIT || tok < a.M) red[(warp * WT + n_local) * a.red_m + tok] = tot[b][f][jj];
          }
    }
    MLD_CONSUMER_BARRIER();
    if (a.ksplit > 1 && pass == 0) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (CUT ? kr > 0 : a.ksplit > 1 && kr == 1) {
      peer_remote = map_to_rank(smem_u32(CUT ? peer + (kr - 1) * WT * a.peer_m : peer), 0);
      bar_remote = map_to_rank(smem_u32(peer_bar), 0);
    }
    if (a.ksplit > 1 && kr == 0) {
      if (!mbar_wait_cluster(peer_bar, pass & 1)) {
        atomicExch(a.error, 3);
        failed = true;
      }
    }
    // the sum of output n_local for a token over the warps that hold a share of it: all of them, or every n_rr-th
    const auto warp_sum = [&](int n_local, int tok) {
      float v = 0.0f;
      if (SPLIT) {
        for (int w = tok >> 3; w < kConsumerWarps; w += n_rr) v += red[(w * WT + n_local) * a.red_m + (tok & 7)];
      } else {
#pragma unroll
        for (int w = 0; w < kConsumerWarps; ++w) v += red[(w * WT + n_local) * a.red_m + tok];
      }
      return v;
    };
    // CUT: the other CTAs' sums of an output onto this one's, in the order of their parts of K
    [[maybe_unused]] const auto add_peers = [&](float v, int n_local, int tok) {
      for (int r = 0; r < partners; ++r) v += peer[(r * WT + n_local) * a.peer_m + tok];
      return v;
    };
    if (CUT ? kr > 0 : a.ksplit > 1 && kr == 1) {
      // a later part of K: hand the sums to the cluster's first CTA
      for (int idx = threadIdx.x; idx < WT * a.M && !failed; idx += kConsumerWarps * 32) {
        const int n_local = idx / a.M, tok = idx - n_local * a.M;
        st_cluster_f32(peer_remote + (n_local * a.peer_m + tok) * 4, warp_sum(n_local, tok));
      }
    } else if (a.epilogue == MLD_EPILOGUE_SWIGLU_PAIRS) {
      // rows alternate gate_i, up_i: out[i] = silu(gate_i) * up_i, each rounded to
      // fp16 where the unfused graph would store it
      for (int idx = threadIdx.x; idx < (WT / 2) * a.M && !failed; idx += kConsumerWarps * 32) {
        const int p_local = idx / a.M, tok = idx - p_local * a.M;
        float sg = warp_sum(2 * p_local, tok), su = warp_sum(2 * p_local + 1, tok);
        if constexpr (CUT) {
          sg = add_peers(sg, 2 * p_local, tok);
          su = add_peers(su, 2 * p_local + 1, tok);
        } else if (a.ksplit > 1) {
          sg += peer[(2 * p_local) * a.peer_m + tok];
          su += peer[(2 * p_local + 1) * a.peer_m + tok];
        }
        const int n = n0 + 2 * p_local;
        if (n + 1 < n_end) {
          const float g = __half2float(__float2half_rn(sg * kOutScale));
          const float u = __half2float(__float2half_rn(su * kOutScale));
          const __half r = __float2half_rn(g / (1.0f + __expf(-g)) * u);
          const int i = n >> 1, tk_out = a.tok0 + tok;
          const int64_t yi = a.dst_layout == MLD_LAYOUT_SLICED ? (((int64_t)(i >> 2) * a.M_total + tk_out) * 4 + (i & 3))
                                                               : ((int64_t)tk_out * (a.N / 2) + i);
          if (a.scatter.world > 1) {
            for (int pr = 0; pr < a.scatter.world; ++pr) static_cast<__half*>(a.scatter.y_peers[pr])[yi] = r;
          } else {
            static_cast<__half*>(a.y)[yi] = r;
          }
        }
      }
    } else {
      for (int idx = threadIdx.x; idx < WT * a.M && !failed; idx += kConsumerWarps * 32) {
        const int n_local = idx / a.M, tok = idx - n_local * a.M;
        const int n = n0 + n_local;
        if (n >= n_end) continue;
        float s = warp_sum(n_local, tok);
        if constexpr (CUT) {
          s = add_peers(s, n_local, tok);
        } else if (a.ksplit > 1) {
          s += peer[n_local * a.peer_m + tok];  // fixed order: lower half of K first
        }
        __half r = __float2half_rn(s * kOutScale);
        if (a.bias != nullptr) r = __hadd(r, static_cast<const __half*>(a.bias)[n]);
        const int tk_out = a.tok0 + tok;
        const int64_t yi = a.dst_layout == MLD_LAYOUT_SLICED ? (((int64_t)(n >> 2) * a.M_total + tk_out) * 4 + (n & 3))
                                                             : ((int64_t)tk_out * a.N + n);
        if (a.dst_layout == MLD_LAYOUT_SLICED || n < a.N) {
          if (a.scatter.world > 1) {
            for (int pr = 0; pr < a.scatter.world; ++pr) static_cast<__half*>(a.scatter.y_peers[pr])[yi] = r;
          } else {
            static_cast<__half*>(a.y)[yi] = r;
          }
        }
      }
    }
    if (CUT ? kr > 0 : a.ksplit > 1 && kr == 1) mbar_arrive_cluster(bar_remote);  // release: the stores above are visible
    MLD_CONSUMER_BARRIER();
    if (tr && threadIdx.x == 0) tr[5] = globaltimer_ns();
  }
  if (a.scatter.world > 1) {
    // every CTA: make its peer stores visible, then count in; the last one
    // raises this rank's flag on every rank
    __threadfence_system();
    MLD_CONSUMER_BARRIER();
    if (threadIdx.x == 0) {
      const int t = atomicAdd(a.scatter.ticket, 1);
      if (t == static_cast<int>(gridDim.x) - 1) {
        *a.scatter.ticket = 0;
        __threadfence_system();
        const unsigned seq = static_cast<unsigned>(*a.scatter.step * a.scatter.seq_per_step + a.scatter.seq_off);
        for (int pr = 0; pr < a.scatter.world; ++pr) st_release_sys(a.scatter.flag_peers[pr], seq);
      }
    }
  }
}

template <int BITS, int W, bool SUBNORMAL, bool MONE, bool DIGITS, bool ZP, bool SPLIT, bool INTERLEAVE, bool CUT = false>
int launch_strip_f(const CUtensorMap& tw, const CUtensorMap& ts, const CUtensorMap& tz, const StripArgs& a,
                   const StripGeometry& gm, cudaStream_t stream) {
  auto kern = fc_strip_kernel<BITS, W, SUBNORMAL, MONE, DIGITS, ZP, SPLIT, INTERLEAVE, CUT>;
  static bool configured[kMaxDevices];  // per instantiation and device
  int dev;
  if (needs_configure(configured, &dev)) {
    MLD_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    if (dev >= 0) configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(gm.grid, 1, 1);
  cfg.blockDim = dim3((kConsumerWarps + 1) * 32, 1, 1);
  cfg.dynamicSmemBytes = gm.smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  int na = 0;
  if (gm.ksplit > 1) {
    attrs[na].id = cudaLaunchAttributeClusterDimension;
    attrs[na].val.clusterDim.x = gm.ksplit;
    attrs[na].val.clusterDim.y = 1;
    attrs[na].val.clusterDim.z = 1;
    ++na;
  }
  if (a.pdl) {
    attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = na;
  MLD_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tw, ts, tz, a));
  count_launch();
  return MLD_OK;
}

template <int BITS, int W, bool SUBNORMAL, bool MONE, bool DIGITS = false, bool ZP = false, bool SPLIT = false>
int launch_strip_t(const CUtensorMap& tw, const CUtensorMap& ts, const CUtensorMap& tz, const StripArgs& a,
                   const StripGeometry& gm, cudaStream_t stream) {
  if constexpr (W == 2 && MONE && !SPLIT) {  // (one token, strips of two whole boxes)
    if (gm.ksplit > 2) return launch_strip_f<BITS, W, SUBNORMAL, MONE, DIGITS, ZP, SPLIT, false, true>(tw, ts, tz, a, gm, stream);
  }
  if (gm.ksplit > 2) {  // (the other forms add up two parts and would drop the rest)
    set_last_error_text("no form of the streaming kernel adds up more than two parts of K for these strips");
    return MLD_UNIMPLEMENTED;
  }
  if constexpr (W == 2) {  // (strips of several passes with pdl are two boxes wide)
    if (!MONE || gm.interleave) return launch_strip_f<BITS, W, SUBNORMAL, MONE, DIGITS, ZP, SPLIT, true>(tw, ts, tz, a, gm, stream);
  }
  if constexpr (W != 2 || MONE) return launch_strip_f<BITS, W, SUBNORMAL, MONE, DIGITS, ZP, SPLIT, false>(tw, ts, tz, a, gm, stream);
}

template <int BITS, int W, bool ZP>
int launch_strip_w(bool subnormal, bool mone, const CUtensorMap& tw, const CUtensorMap& ts, const CUtensorMap& tz,
                   const StripArgs& a, const StripGeometry& gm, cudaStream_t stream) {
  if constexpr (W <= 2) {
    if constexpr (!ZP) {
      if (gm.ts_shift > 0 && !subnormal) return launch_strip_t<BITS, W, false, false, false, false, true>(tw, ts, tz, a, gm, stream);
    }
    if (gm.ts_shift > 0) return launch_strip_t<BITS, W, true, false, false, ZP, true>(tw, ts, tz, a, gm, stream);
  }
  if (ZP || subnormal) {
    if constexpr (!ZP) {
      if (gm.xdig_bytes > 0) return launch_strip_t<BITS, W, true, true, true>(tw, ts, tz, a, gm, stream);
    }
    if (mone) return launch_strip_t<BITS, W, true, true, false, ZP>(tw, ts, tz, a, gm, stream);
    return launch_strip_t<BITS, W, true, false, false, ZP>(tw, ts, tz, a, gm, stream);
  }
  if constexpr (!ZP) {
    if (mone) return launch_strip_t<BITS, W, false, true>(tw, ts, tz, a, gm, stream);
    return launch_strip_t<BITS, W, false, false>(tw, ts, tz, a, gm, stream);
  }
  set_last_error_text("zero points take the subnormal operand form");
  return MLD_INVALID_ARGUMENT;
}

}  // namespace

StripGeometry strip_geometry(int bits, int N, int K, int m_total, int group_slices, int scale_mode, int sms,
                             bool pdl, int smem_limit_kb, bool zero_point, bool split) {
  StripGeometry gm;
  memset(&gm, 0, sizeof gm);
  // tokens per launch: an MMA's eight, or up to four times that where the warps can split them
  gm.launch_tokens = split && pdl ? kStripTokens : 8;
  gm.ts_shift = gm.launch_tokens == 8 ? 0 : m_total > 16 ? 2 : m_total > 8 ? 1 : 0;
  const int N4 = align_n(N, 4), SS = div_up(K, 4);
  const int box_n = bits == 4 ? 64 : 32;
  const int row_bytes = (N4 / 4) * (bits == 4 ? 8 : 16);
  gm.gran = bits == 4 ? 1 : 2;
  const int C = row_bytes / 16;
  gm.units = C / gm.gran;
  // Overlapping launches need two CTAs per SM, which the register file grants to the instantiations of up
  // to two boxes per stage: wider strips take more column passes instead.
  const int w_max = pdl ? 2 : 4;
  // Two CTAs per strip (a cluster splitting K) when single strips would be
  // narrower than 128 bytes and K is long enough to halve.
  gm.ksplit = (C < 8 * sms && SS >= 4 * kStageRows && sms >= 2) ? 2 : 1;
  int strips = sms / gm.ksplit;
  if (gm.ksplit == 1 && w_max <= 2 && C > 8 * w_max * sms) {
    // More columns than one pass of one CTA per SM: two CTAs share each SM, so that one streams while the other is in a
    // pass's epilogue (151936 x 2048 INT8, one token, fp16 form: 17 passes of a lone CTA 85.8 us, 9 of two 69.7; with the
    // passes of all strips side by side 64.0, against 47.6 for the bytes at the copy rate).
    strips = 2 * sms;
    gm.interleave = C > 8 * w_max * strips ? 1 : 0;
  }
  if (strips > gm.units) strips = gm.units;
  if (strips < 1) strips = 1;
  gm.strips = strips;
  gm.grid = strips * gm.ksplit;
  int max_width = div_up(gm.units, strips) * gm.gran;  // chunks
  int w = div_up(max_width, 8);
  if (gm.ksplit > 1 && w > w_max) {  // a cluster pair runs a single pass
    gm.ksplit = 1;
    strips = sms < gm.units ? sms : gm.units;
    gm.strips = strips;
    gm.grid = strips;
    max_width = div_up(gm.units, strips) * gm.gran;
    w = div_up(max_width, 8);
  }
  // One token: strips that fill their boxes, where the rule above leaves part of them empty or splits what is small already.
  // us in a graph, INT4 block 32 unless said otherwise, the rule above / as here.
  if (m_total == 1 && w_max == 2) {
    const int n_st = div_up(SS, kStageRows), most = sms + sms * 73 / 100;
    int S = 0, boxes = 2;
    if (C < 8 * sms && n_st <= 8) {
      // up to 2048 inputs the stages of a whole strip take less time than the cluster's meeting: 2048 x 4096 4.5 / 4.3,
      // 1024 x 3072 4.0 / 3.4, 1024 x 1024 4.0 / 3.0 (4096 x 4096, on the other side of the line: 5.5 / 6.5)
      S = 1;
      boxes = 1;
    } else if (C <= 16 * most) {
      // Strips of two whole boxes.  As many as SMs or more, or K cut so that a CTA has up to eight stages (it also turns that
      // much of the vector into digits) where clusters of that size are all resident at once and every SM has work: 4096 x
      // 11008 10.0 / 9.0 (2 x 86 CTAs; 3 x 86 9.2), 4096 x 14336 10.0 / 9.5, 14336 x 4096 12.9 / 10.3,
      // 4096 x 22016 14.8 / 13.1, 1536 x 21568 8.9 / 6.7, INT8 4096 x 11008 13.9 / 12.8.  On the other side of the
      // line: clusters of three (4736 x 8320 7.6 / 8.7), fewer than sixteen stages to cut (INT8 2432 x 6048 6.0 / 6.4) and
      // idle SMs (2048 x 16384 6.2 / 7.6).
      // (Only where strips reach into their second box: the form for more than two parts has two.)
      // More than two parts only where the rule above fills its boxes badly for the number of stages that there are to share out:
      // smaller parts and the longer meeting cost more than empty chunks in short strips (per cent of the boxes filled:
      // 4608 x 8192 86 7.9 / 8.9, INT8 4608 x 3072 65 6.6 / 7.2, INT8 6144 x 4096 86 8.2 / 9.3, 8704 x 4584 97 8.2 / 8.8; on the other side
      // 6144 x 5120 54 8.9 / 7.9, 10240 x 5120 54 13.1 / 9.8, 14336 x 4096 86 12.9 / 10.3, 16384 x 4608 97 14.4 / 13.0).
      const int full = div_up(C, 16), filled = 100 * C / (strips * w * 8);
      const int line = n_st >= 60 ? 100 : n_st >= 40 ? 90 : 2 * n_st + 10;
      if (full >= sms) {
        S = 1;
      } else if (n_st >= 16 && C > 8) {
        for (int s = 2; s <= 8 && full * s <= most; ++s) {
          if (s == 3) continue;
          S = s;
          if (div_up(n_st, s) <= 8) break;
        }
        if (full * S < sms || (S > 2 && filled > line)) S = 0;
      }
    }
    if (S > 0) {
      gm.interleave = 0;
      gm.ksplit = S;
      gm.strips = strips = div_up(C, 8 * boxes);
      gm.grid = strips * S;
      max_width = div_up(gm.units, strips) * gm.gran;
      w = div_up(max_width, 8);
    }
  }
  gm.w = w > w_max ? w_max : w;
  const int passes = gm.interleave ? div_up(C, strips * gm.w * 8) : div_up(max_width, gm.w * 8);
  gm.fill = 100 * C / (strips * passes * gm.w * 8);
  gm.rows_per_split = align_n(div_up(SS, gm.ksplit), kStageRows);
  if (scale_mode == MLD_SCALE_SCALAR) {
    gm.scale_rows = 0;
    gm.group_slices = 1;
    gm.gs_shift = -1;
  } else {
    gm.group_slices = scale_mode == MLD_SCALE_PER_CHANNEL ? align_n(SS, kStageRows) : group_slices;
    gm.scale_rows = gm.group_slices >= kStageRows ? 1 : kStageRows / gm.group_slices;
    gm.gs_shift = -1;
    if (gm.group_slices < kStageRows)
      for (int sh = 3; sh < 7; ++sh)
        if ((1 << sh) == gm.group_slices) gm.gs_shift = sh;
  }
  const int wt = gm.w * box_n;
  gm.zp_off = align_n(gm.scale_rows * wt * 2, 128);
  gm.scale_stage_bytes = zero_point ? 2 * gm.zp_off : gm.zp_off;
  const int x_bytes = align_n(kStageRows * m_total * 8, 128);
  gm.stage_bytes = align_n(gm.w * kBoxBytes + gm.scale_stage_bytes + x_bytes, 1024);
  gm.red_m = m_total < 8 ? m_total : 8;
  gm.peer_m = gm.ksplit == 1 ? 0 : m_total < gm.launch_tokens ? m_total : gm.launch_tokens;
  gm.stage_rows = kStageRows;
  // With programmatic dependent launch two consecutive GEMVs share an SM while
  // one drains and the next prefetches, so each takes at most half of it.
  int budget = pdl ? 112 * 1024 : 224 * 1024;
  if (smem_limit_kb >= 32 && smem_limit_kb <= 224) budget = smem_limit_kb * 1024;
  int fixed = (kConsumerWarps * gm.red_m + (gm.ksplit - 1) * gm.peer_m) * wt * 4 + 8 + (2 * 16 + 1) * 8 + 1024 + 64;
  // One token as digits: room for the activation vector of this CTA's K range (per k-slice 8 bytes, 4 digits 16 more; per
  // unit of eight k-slices 8 bytes for every two digits; a barrier).
  if (m_total == 1 && split && !zero_point) {
    const int xdig = gm.rows_per_split * (bits == 4 ? 9 : 26) + 48;
    if (bits == 4) {
      gm.xdig_bytes = xdig;
    } else {
      // 8-bit weights take four digits where a CTA multiplies enough by them to pay for turning the whole vector into them,
      // and only as long as the ring keeps three stages beside them.  us in a graph, fp16 form / digits: 151936 x 2048 55.8 /
      // 49.1, 65536 x 2048 28.1 / 24.8, 12288 x 4096 14.8 / 13.8, 12288 x 8192 27.7 / 25.4; below the first line 12288 x 1024
      // 6.0 / 6.4, 32000 x 640 7.5 / 8.1, 8192 x 4096 9.4 / 9.9; below the second 16384 x 11008 36.6 / 42.9.
      const bool pays = strips > sms && passes * (gm.rows_per_split / kStageRows) >= 16;
      gm.xdig_bytes = pays && (budget - fixed - xdig) / gm.stage_bytes >= 3 ? xdig : 0;
    }
    fixed += gm.xdig_bytes;
  }
  int stages = (budget - fixed) / gm.stage_bytes;
  if (stages > 16) stages = 16;
  if (stages < 2) stages = (227 * 1024 - fixed) / gm.stage_bytes;
  gm.stages = stages;
  gm.smem_bytes = (size_t)stages * gm.stage_bytes + fixed;
  return gm;
}

int launch_fc_strip(int bits, bool subnormal, const CUtensorMap& tw, const CUtensorMap& ts, const CUtensorMap* tz,
                    const StripArgs& a, const StripGeometry& gm, cudaStream_t stream) {
  if (a.M == 0 || gm.grid == 0) return MLD_OK;
  const bool mone = a.M == 1;
#define MLD_W(B, WV) \
  case WV:           \
    return launch_strip_w<B, WV, false>(subnormal, mone, tw, ts, tw, a, gm, stream)
#define MLD_WZ(B, WV) \
  case WV:            \
    return launch_strip_w<B, WV, true>(subnormal, mone, tw, ts, *tz, a, gm, stream)
  if (tz != nullptr) {  // (zero points are taken with pdl only, whose strips have two boxes at most)
    if (bits == 4) {
      switch (gm.w) {
        MLD_WZ(4, 1);
        MLD_WZ(4, 2);
      }
    } else {
      switch (gm.w) {
        MLD_WZ(8, 1);
        MLD_WZ(8, 2);
      }
    }
  } else if (bits == 4) {
    switch (gm.w) {
      MLD_W(4, 1);
      MLD_W(4, 2);
      MLD_W(4, 3);
      MLD_W(4, 4);
    }
  } else {
    switch (gm.w) {
      MLD_W(8, 1);
      MLD_W(8, 2);
      MLD_W(8, 3);
      MLD_W(8, 4);
    }
  }
#undef MLD_W
#undef MLD_WZ
  set_last_error_text("bad strip geometry");
  return MLD_INVALID_ARGUMENT;
}

}  // namespace mld
