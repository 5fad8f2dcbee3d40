// Prefill-stage dequant-GEMM with the dequantised weights in TENSOR MEMORY, on pairs of SMs
// (tcgen05 cta_group::2, A operand from tensor memory).
//
// Same contract as gemm_pair_kernel's inline modes (the packed weights never leave their reference layout in
// HBM; arithmetic of the WeightsConverter, ml_drift/common/kernels/conv_weights_converter.cc:248-290, followed
// by an fp16 x fp16 -> fp32 product as the float convolution of common/gpu_model_builder.cc:1110-1276 computes
// it), but with the operand roles turned round:
//
//   Y^T[N x M] = W[N x K] X[M x K]^T
//
// With int8 activations (quantised per token by the kernel ahead) the weights go to tensor memory as signed bytes, exact
// products are summed in int32, and the epilogue dequantises them.  8192 -> 3584, in a graph: 17 tokens 21 us (62 through
// shared memory, 44 with a conversion pass), 512 46 (70, 51), 2048 92 (127, 96).
//
// The weights are the MMA's M-side operand and sit in tensor memory; the activations are the N-side operand in
// shared memory.  A dequantised weight tile is then written once, by tcgen05.st, into the memory the tensor
// core reads it from, instead of being written to shared memory by the transform warps and read back from
// there by the tensor core beside their own traffic - which is what held gemm_pair_kernel's inline modes at
// about 1000 cycles per 64-wide K stage against 560 with prepared operands.
//
// A cluster of two CTAs owns a tile of 256 output channels x tile_tok tokens (tile_tok <= 256).  Per CTA:
//   warp 0       TMA producer of the activation tiles: this CTA's half of the tile's tokens, K-major rows of
//                128 bytes in the 128-byte swizzle, eight stages
//   warp 22      TMA producer of the packed weight boxes ([K/4] rows of 4x4 blocks) of this CTA's 128 channels
//   warps 6..21  transform: four groups of four warps on every fourth stage; a thread owns one output channel
//                (= one TMEM lane; a warp can only address the lane quarter 32 * (warp % 4)), dequantises the
//                stage's 64 input channels to 32 registers of two halves and stores them to the stage's 32
//                tensor-memory columns.  (Bound by the instructions that all warps issue: with eight warps to a
//                stage, half the channels each, a third of them went into what a stage costs a warp anyway.)
//   warp 1       tensor-memory owner; in the first CTA also the MMA issuer: four tcgen05.mma per stage (K = 16
//                each, A = 8 TMEM columns, B = 32 bytes further into the swizzled rows)
//   warps 2..5   epilogue: a thread reads its output channel's accumulators (one TMEM lane, a column per token),
//                adds the bias, and four neighbouring lanes exchange values so that each holds the four channels
//                of one output slice for two tokens, a 16-byte piece of the sliced output layout
// Tensor memory: columns 0..255 accumulators (one buffer: reading a tile's accumulators is not overlapped with
// the next tile's MMAs, so the transform warps share the reading with the epilogue warps; a CTA that works
// alone has two buffers of 128), columns 256..511 the weight ring (8 stages x 32 columns).
// The split of the work over the pairs (tiles of the last wave shared along K) is gemm_pair_kernel's.
// Every wait is bounded.
#include <cuda_fp16.h>

#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "pair_common.cuh"

namespace mld {
namespace {

constexpr int kWtStages = 8;          // operand ring: activation tile in shared memory + weight tile in TMEM
constexpr int kWtRows = 128;          // output channels per CTA
constexpr int kWtTokBytes = 128 * kKBytes;  // up to 128 token rows per CTA and stage
constexpr uint32_t kWtACol = 256;     // first TMEM column of the weight ring
constexpr int kWtAccCols = 128;       // columns of each of a lone CTA's two sets of accumulators
constexpr int kErrWtBase = 50;
constexpr int kXfWarps = 4;            // transform warps that share a stage, one per quarter of the channels
constexpr int kDrainParts = 5;        // warps that read one lane quarter's accumulators: one epilogue + four transform

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// D[tmem_d] (+)= A[tmem_a] B[desc_b]^T over the pair (or by this CTA alone); A: 16 halves per lane in 8 columns of
// tensor memory (of both CTAs').
template <bool PAIR, bool I8>
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                        uint32_t accumulate) {
  if constexpr (PAIR && I8) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], [%1], %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
  } else if constexpr (I8) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
  } else if constexpr (PAIR) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
  }
}
// Arrives on a barrier of the pair's first CTA.  What it orders is tensor memory, by tcgen05.wait and
// fence::before_thread_sync ahead of it; releasing at cluster scope on top of that would take about 800 cycles.
__device__ __forceinline__ void arrive_in_pair(uint32_t cluster_addr, uint32_t n = 1) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_addr), "r"(n) : "memory");
}
// Arrives on the barrier (in both CTAs of a pair) once every MMA issued so far has completed.
template <bool PAIR>
__device__ __forceinline__ void commit(uint64_t* bar) {
  if constexpr (PAIR) {
    commit_pair(bar);
  } else {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
  }
}
template <bool PAIR>
__device__ __forceinline__ void tmem_alloc_all(uint32_t* smem_dst) {
  if constexpr (PAIR) {
    tmem_alloc_pair(smem_dst, 512);
    tmem_relinquish_pair();
  } else {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(smem_dst)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
}
template <bool PAIR>
__device__ __forceinline__ void tmem_dealloc_all(uint32_t taddr) {
  if constexpr (PAIR) {
    tmem_dealloc_pair(taddr, 512);
  } else {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(taddr) : "memory");
  }
}

// (1024 + u) - (1024 + zero) is exact, so the dequantised weight is rounded once.  (The WeightsConverter rounds u s, zero s
// and their difference, which is further from (u - zero) s and an instruction more.)
__device__ __forceinline__ uint32_t dq_once(uint32_t biased, __half2 offset, __half2 s2) {
  const __half2 r = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&biased), offset), s2);
  return *reinterpret_cast<const uint32_t*>(&r);
}

// The piece after pc in a share of every `parts`-th unit of `unit` (1 or 2) pieces.
__device__ __forceinline__ int next_piece(int pc, int unit, int parts) {
  return unit == 2 && (pc & 1) == 0 ? pc + 1 : pc + 1 + (parts - 1) * unit;
}

struct WtArgs {
  PairArgs p;       // M, N, N4, k_blocks, scales, bias, y, dst_layout, error, outs, split, work list, w ring
  int tile_tok;     // tokens per tile (UMMA N), a multiple of 16
  int tok_tiles;    // ceil(M / tile_tok)
  long long* trace; // tuning builds only: [grid][8] cycle counts
  int trace_flags;  // tuning builds only: 1 = no output stores, 2 = no lane exchange either
};

// PAIR: the two-CTA form described above.  Otherwise a CTA works alone on tiles of 128 output channels x up to 128
// tokens: twice as many, smaller tiles, at the price of every CTA fetching all of the tile's tokens.
// Bound by the transformation (64 x 128 weights a stage and CTA at five instructions for two) beside whatever else the warps
// issue: a pair's stage takes about 700 cycles, 512 of them its MMAs; a lone CTA's MMAs need 160 to 260.
// 4096 x 11008 INT4, in a graph: 77 tokens 23.0 us (30.5 with eight warps to a stage and one set of accumulators, 41.1 with
// pairs and whole tiles); 256 tokens 31.0, 512 45.6 (34.2, 48.5 with all five warps of a quarter reading the sums that are
// handed over; 42.9, 66.7 with stages announced to the pair's first CTA by warps of their own as well, whose release at
// cluster scope took longer than a stage).
constexpr int kWtThreads = 23 * 32;
template <int MODE>
constexpr int kWtSlices = MODE == kModeInt8I8 ? 32 : 16;

// The bytes of two 4x4 blocks turned round over the four lanes c = 0..3 that share them: lane c comes with word c (input
// channel c, a byte per output) of each and leaves with output c's bytes of the four input channels, as signed numbers.
// Two butterfly steps (lanes 2 apart, then 1), both blocks' halves in one shuffle.  (A lane reading whole blocks, of which
// it needs a quarter, would take the shared memory twice the time of word and shuffle.)
struct TurnSelectors {
  uint32_t give2, keep2, give1, keep1, out0, out1;
  __device__ __forceinline__ explicit TurnSelectors(int c) {
    // step 1: bytes of outputs 2h, 2h + 1 stay with the lanes whose c / 2 is h
    keep2 = (c & 2) ? 0x7632u : 0x5410u;
    give2 = (c & 2) ? 0x5410u : 0x7632u;
    // step 2, of {own, received}: bytes {block 0 own, block 0 received, block 1 own, block 1 received} of output c (c ^ 1)
    keep1 = (c & 1) ? 0x7351u : 0x6240u;
    give1 = (c & 1) ? 0x6240u : 0x7351u;
    // then {kept, received} hold input channels c, c ^ 2 and c ^ 1, c ^ 3: in the order of the channels
    uint32_t s = 0;
    for (int k = 0; k < 4; ++k) s |= static_cast<uint32_t>(k == c ? 0 : k == (c ^ 2) ? 1 : k == (c ^ 1) ? 4 : 5) << (4 * k);
    out0 = s;
    out1 = s + 0x2222u;
  }
};
__device__ __forceinline__ void turn_blocks(uint32_t w0, uint32_t w1, const TurnSelectors& t, uint32_t& o0, uint32_t& o1) {
  const uint32_t k2 = __byte_perm(w0, w1, t.keep2), r2 = __shfl_xor_sync(0xffffffffu, __byte_perm(w0, w1, t.give2), 2);
  const uint32_t k1 = __byte_perm(k2, r2, t.keep1), r1 = __shfl_xor_sync(0xffffffffu, __byte_perm(k2, r2, t.give1), 1);
  o0 = __byte_perm(k1, r1, t.out0) ^ 0x80808080u;
  o1 = __byte_perm(k1, r1, t.out1) ^ 0x80808080u;
}
template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kWtThreads, 1)
    gemm_wtmem_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, WtArgs wa) {
  const PairArgs& a = wa.p;
  constexpr bool I8 = MODE == kModeInt8I8;
  constexpr int BLK = MODE == kModeInt4F16 ? 8 : 16;   // bytes of a packed 4x4 block
  constexpr int SLICES = kWtSlices<MODE>;               // packed rows per stage (64 input channels, 128 of a byte)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int CTAS = PAIR ? 2 : 1;                    // CTAs per tile
  const int cta_tok = wa.tile_tok / CTAS;               // token rows this CTA fetches
  constexpr int w_pitch = (kWtRows / 4) * BLK;          // bytes of one packed row of the box
  constexpr int w_stage = SLICES * w_pitch;             // 4 / 8 / 16 KB
  uint8_t* sX = smem;
  uint8_t* sW = sX + (size_t)kWtStages * kWtTokBytes;
  uint64_t* full_w = reinterpret_cast<uint64_t*>(sW + (size_t)a.w_stages * w_stage);  // [w_stages]
  uint64_t* w_empty = full_w + a.w_stages;            // [w_stages]: the transform warps have read the box
  uint64_t* full_ab = w_empty + a.w_stages;           // [stages], first CTA: tokens of both CTAs landed, weights of both in TMEM
  uint64_t* empty = full_ab + kWtStages;              // [stages]: the stage's MMAs have completed (arrives in both CTAs)
  uint64_t* tmem_full = empty + kWtStages;            // [3] (see accumulators_ready), arrives in both CTAs
  uint64_t* tmem_empty = tmem_full + 3;               // [2], first CTA: the warps that read it (of both CTAs) are done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_rank() : 0u;
  // ("pair": whoever works on a tile; numbered backwards, so that the pairs another one waits for began before it)
  const int n_pairs = gridDim.x / CTAS, pair = n_pairs - 1 - static_cast<int>(blockIdx.x) / CTAS;
  WorkList work0;
  {
    const int shared_units = a.shared_tiles * a.k_blocks;
    work0.u = min(shared_units, pair * a.units_per_pair);
    work0.u_end = min(shared_units, work0.u + a.units_per_pair);
    work0.tile = a.shared_tiles + pair;
    work0.tile_end = a.m_tiles * a.n_tiles;
    work0.tile_step = n_pairs;
    work0.k_blocks = a.k_blocks;
  }

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.w_stages; ++s) {
      mbar_init(&full_w[s], 1);
      mbar_init(&w_empty[s], kXfWarps);
    }
    for (int s = 0; s < kWtStages; ++s) {
      mbar_init(&full_ab[s], 1 + CTAS * kXfWarps);  // the producer's expect_tx, the transform warps
      mbar_init(&empty[s], 1);
    }
    mbar_init(&tmem_full[2], 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], PAIR ? CTAS * 4 * kDrainParts : 4);
    }
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc_all<PAIR>(tmem_slot);
  tc_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();  // the partner's barriers are initialised before anything arrives on them
  tc_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t full_ab_lead = PAIR ? map_shared(smem_u32(full_ab), 0) : 0u;
  const uint32_t tmem_empty_lead = PAIR ? map_shared(smem_u32(tmem_empty), 0) : 0u;
  // (a pair's accumulators are read by five warps of a quarter or by one, which then arrives for all)
  auto release_tmem = [&](int part, int parts, int acc) {
    if constexpr (PAIR)
      arrive_in_pair(tmem_empty_lead, kDrainParts / parts);
    else if (part == 0)
      mbar_arrive(&tmem_empty[acc]);
  };
  // tile -> (token tile, channel tile): the token tiles of one channel tile follow each other
  auto tile_tok0 = [&](int tile) { return (tile % a.m_tiles) * wa.tile_tok; };
  auto tile_n0 = [&](int tile) { return (tile / a.m_tiles) * CTAS * kWtRows; };

  // Who reads a segment's accumulators: the quarter's epilogue warp alone, while the transform warps go on with the next
  // tile, or all five warps that can address the quarter.  A lone CTA has a second set of accumulators, so that its MMAs go
  // on, too: all join in for the last segment only.  A pair's MMAs wait for the reading, and the ring holds eight stages: one
  // warp does for the raw sums that are handed over, but with whole tiles it takes longer than all five (4096 x 14336, 1024
  // tokens 93.5 us against 86.8; 256 tokens, a handed-over part and a last one: 33.4 against 36.4).
  const auto read_by_all = [&](const Segment& sg, bool last) { return last || (PAIR && sg.kb0 == 0); };
  // The barrier that a segment's finished MMAs arrive on.  A wait tells one use of a barrier from the one before and no more, so
  // nobody may miss a use of one that it waits on later: segments that the epilogue warp reads alone have barriers that it
  // alone waits on, by accumulators, and those read by all have the third.  (With a segment of a few stages a transform
  // warp is done while the MMAs of segments before it are still to come, since the ring holds eight stages.)
  const auto accumulators_ready = [&](const Segment& sg, bool last, int nth) {
    return &tmem_full[read_by_all(sg, last) ? 2 : PAIR ? 0 : nth & 1];
  };

  // Accumulators -> outputs, the share `part` of `parts` of those warps: pieces of 16 token columns, every parts-th (pairs:
  // two together).
  // A tile cut along K: a pair (CTA) whose share does not begin with the tile's first k-block (always the first of its
  // segments, so that nothing it waits for comes before) leaves its raw accumulators in its own workspace slot; the one that
  // has the first k-block adds the following slots to its own accumulators, in order, and writes the outputs.  Blocks begin
  // in the order of their numbers, so those it waits for hold SMs already, whatever else is on the GPU.  A slot has a flag
  // per lane quarter and piece (two pieces), since its writer and reader may be shared differently.
  auto drain = [&](const Segment& sg, int part, int parts, int acc) -> bool {
    const int quad = warp & 3;  // TMEM lanes 32*quad .. 32*quad+31 belong to this warp
    const bool hands_over = sg.kb0 > 0, takes_over = !hands_over && sg.kb1 < a.k_blocks;
    const auto rows_of = [&](int slot) {
      return reinterpret_cast<uint4*>(a.split_ws) + ((size_t)(slot * CTAS + static_cast<int>(rank)) * 4 + quad) * (8 * 8 * 32) + lane;
    };
    const auto flag_of = [&](int slot, int i) {  // the i-th flag that this warp's share has
      return a.split_flags + ((slot * CTAS + static_cast<int>(rank)) * 4 + quad) * 8 + part + i * parts;
    };
    // the pairs that hold the rest of a tile this pair completes
    const int others = takes_over ? ((sg.tile + 1) * a.k_blocks - 1) / a.units_per_pair - pair : 0;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(PAIR ? 0 : acc * kWtAccCols);
    constexpr int kUnit = PAIR ? 2 : 1;  // pieces that go together: a quarter has eight flags
    const int n_pieces = wa.tile_tok >> 4;
    const int n_units = (n_pieces + kUnit - 1) / kUnit, n_flags = part < n_units ? (n_units - part + parts - 1) / parts : 0;
    if (hands_over) {
      uint4* const slot_rows = rows_of(pair);
      for (int pc = kUnit * part; pc < n_pieces; pc = next_piece(pc, kUnit, parts)) {
        uint32_t r[16];
        tmem_ld16(lane_base + static_cast<uint32_t>(16 * pc), r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j) slot_rows[(pc * 4 + j) * 32] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
      }
      __threadfence();
      tc_before();
      __syncwarp();
      if (lane < n_flags) st_release_gpu(flag_of(pair, lane), a.epoch);
      if (lane == 0) release_tmem(part, parts, acc);
      return true;
    }
    if (takes_over) {
      bool seen = true;
      for (int i = lane; i < others * n_flags; i += 32) {  // a lane per flag
        const uint32_t* flag = flag_of(pair + 1 + i / n_flags, i % n_flags);
        const unsigned long long t0 = globaltimer_ns();
        uint32_t v;
        while ((v = ld_acquire_gpu(flag)) != a.epoch && globaltimer_ns() - t0 <= kWaitLimitNs) __nanosleep(32);
        seen = seen && v == a.epoch;
      }
      if (!__all_sync(0xffffffffu, seen)) {
        atomicExch(a.error, kErrWtBase + 8);
        return false;
      }
      // each flag has this one reader, which takes it back: a replayed graph launches with the same epoch again
      for (int i = lane; i < others * n_flags; i += 32) __stcg(flag_of(pair + 1 + i / n_flags, i % n_flags), 0u);
    }
    const int n = tile_n0(sg.tile) + static_cast<int>(rank) * kWtRows + quad * 32 + lane;  // output channel
    const int m_first = (sg.tile % a.m_tiles) * wa.tile_tok;
    const bool has_n = n < a.N4;
    __half bias_h = __float2half_rn(0.0f);
    if (a.bias != nullptr && has_n) bias_h = static_cast<const __half*>(a.bias)[n];
    [[maybe_unused]] float w_scale = 0.0f, w_offset = 0.0f;  // int8 route: the channel's scale, the sum of its weights
    if constexpr (I8) {
      pdl_wait();  // (the tokens' parameters come from the kernel ahead; over by now, whoever waited first)
      if (n < a.N) {
        w_scale = __half2float(a.scale[n]);
        if (a.w_sum != nullptr) w_offset = static_cast<float>(a.w_sum[n]);
      }
    }
    const int q = lane & 3;  // place among the four channels of the output slice n >> 2
    for (int pc = kUnit * part; pc < n_pieces; pc = next_piece(pc, kUnit, parts)) {
      const int c0 = 16 * pc;
      uint32_t r[16];
      tmem_ld16(lane_base + static_cast<uint32_t>(c0), r);
      tmem_ld_wait();
#pragma unroll 2
      for (int o = 0; o < others; ++o) {
        const uint4* const slot_rows = rows_of(pair + 1 + o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 v = __ldcg(&slot_rows[(pc * 4 + j) * 32]);
          if constexpr (I8) {
            r[4 * j] += v.x, r[4 * j + 1] += v.y, r[4 * j + 2] += v.z, r[4 * j + 3] += v.w;
          } else {
            r[4 * j] = __float_as_uint(__uint_as_float(r[4 * j]) + __uint_as_float(v.x));
            r[4 * j + 1] = __float_as_uint(__uint_as_float(r[4 * j + 1]) + __uint_as_float(v.y));
            r[4 * j + 2] = __float_as_uint(__uint_as_float(r[4 * j + 2]) + __uint_as_float(v.z));
            r[4 * j + 3] = __float_as_uint(__uint_as_float(r[4 * j + 3]) + __uint_as_float(v.w));
          }
        }
      }
      if constexpr (I8) {
        // CreateDequantization (quantize_and_dequantize.cc:867-964):
        //   res = float(acc) * (w_scale * src_scale) + w_scale * src_zero_point * weights_sum
        // lanes 0..15 hold the scales of the piece's tokens, 16..31 their zero points
        const int tok = m_first + c0 + (lane & 15);
        const float mine = tok < a.M ? a.a_params[tok * 3 + (lane >> 4)] : 0.0f;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float a_scale = __shfl_sync(0xffffffffu, mine, j), a_off = __shfl_sync(0xffffffffu, mine, 16 + j);
          float v = static_cast<float>(static_cast<int32_t>(r[j])) * (w_scale * a_scale);
          if (a.w_sum != nullptr) v += w_scale * a_off * w_offset;
          r[j] = __float_as_uint(v);
        }
      }
      // token pairs as packed halves: h2[i] = tokens c0 + 2i, c0 + 2i + 1 of channel n
      uint32_t h2[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        __half2 v = __floats2half2_rn(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
        if (a.bias != nullptr) v = __hadd2(v, __half2half2(bias_h));
        h2[i] = *reinterpret_cast<const uint32_t*>(&v);
      }
      if (a.dst_layout == MLD_LAYOUT_SLICED) {
        // Eight tokens at a time: the four lanes of a slice exchange token pairs so that lane q holds tokens
        // 2q, 2q + 1 (of the eight) of all four channels, 16 contiguous bytes of [slice][token][4 channels].
#pragma unroll
        for (int grp = 0; grp < 2; ++grp) {
          // 4 x 4 transpose over the slice's four lanes in two butterfly steps (lanes 2 apart, then 1 apart):
          // lane q starts with its channel's pairs p0..p3 and ends with pair q of channels 0..3
          uint32_t x0 = h2[4 * grp], x1 = h2[4 * grp + 1], x2 = h2[4 * grp + 2], x3 = h2[4 * grp + 3];
          {
            const bool up = (q & 2) != 0;
            const uint32_t s0 = up ? x0 : x2, s1 = up ? x1 : x3;  // what the lane 2 away needs
            const uint32_t r0 = __shfl_xor_sync(0xffffffffu, s0, 2), r1 = __shfl_xor_sync(0xffffffffu, s1, 2);
            if (up) {
              x0 = r0;
              x1 = r1;
            } else {
              x2 = r0;
              x3 = r1;
            }
          }
          {
            const bool up = (q & 1) != 0;
            const uint32_t s0 = up ? x0 : x1, s1 = up ? x2 : x3;  // what the lane 1 away needs
            const uint32_t r0 = __shfl_xor_sync(0xffffffffu, s0, 1), r1 = __shfl_xor_sync(0xffffffffu, s1, 1);
            if (up) {
              x0 = r0;
              x2 = r1;
            } else {
              x1 = r0;
              x3 = r1;
            }
          }
          const int m = m_first + c0 + 8 * grp + 2 * q;  // first of this lane's two tokens
          uint4 pk;
          pk.x = __byte_perm(x0, x1, 0x5410);  // token m: channels 0, 1
          pk.y = __byte_perm(x2, x3, 0x5410);  //          channels 2, 3
          pk.z = __byte_perm(x0, x1, 0x7632);  // token m + 1
          pk.w = __byte_perm(x2, x3, 0x7632);
          if (has_n && m < a.M) {
            const size_t at = ((size_t)(n >> 2) * a.M + m) * 4;  // in halves
            const bool both = m + 1 < a.M && ((at * 2) & 15) == 0;
            const int world = a.outs.world > 1 ? a.outs.world : 1;
            for (int pr = 0; pr < world; ++pr) {
              __half* base = static_cast<__half*>(a.outs.world > 1 ? a.outs.y[pr] : a.y) + at;
              if (both) {
                *reinterpret_cast<uint4*>(base) = pk;
              } else {
                *reinterpret_cast<uint2*>(base) = make_uint2(pk.x, pk.y);
                if (m + 1 < a.M) *reinterpret_cast<uint2*>(base + 4) = make_uint2(pk.z, pk.w);
              }
            }
          }
        }
      } else if (n < a.N) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int m = m_first + c0 + 2 * i;
          if (m < a.M) static_cast<__half*>(a.y)[(size_t)m * a.N + n] = __ushort_as_half(static_cast<unsigned short>(h2[i] & 0xFFFFu));
          if (m + 1 < a.M)
            static_cast<__half*>(a.y)[(size_t)(m + 1) * a.N + n] = __ushort_as_half(static_cast<unsigned short>(h2[i] >> 16));
        }
      }
    }
    tc_before();
    __syncwarp();
    if (lane == 0) release_tmem(part, parts, acc);
    return true;
  };

  if (warp == 0) {
    // ------------------------------------------------ producer of the activation tiles
    if (lane == 0) prefetch_tmap(&tmap_x);
    // Everything else that this kernel reads was complete when the transposition ahead of it let it begin.
    pdl_wait();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    WorkList work = work0;
    Segment sg;
    while (ok && work.next(sg)) {
      const int m0 = tile_tok0(sg.tile) + static_cast<int>(rank) * cta_tok;
      for (int kb = sg.kb0; kb < sg.kb1; ++kb) {
        if (!__all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1))) {
          if (lane == 0) atomicExch(a.error, kErrWtBase + 1);
          ok = false;
          break;
        }
        if (elect_one()) {
          if (rank == 0) mbar_arrive_expect_tx(&full_ab[stage], static_cast<uint32_t>(wa.tile_tok) * kKBytes);
          if constexpr (PAIR)
            tma_load_2d_pair(sX + (size_t)stage * kWtTokBytes, &tmap_x, full_ab_lead + stage * 8, kb * 4 * SLICES, m0);
          else
            tma_load_2d(sX + (size_t)stage * kWtTokBytes, &tmap_x, &full_ab[stage], kb * 4 * SLICES, m0);
        }
        __syncwarp();
        if (++stage == kWtStages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------- MMA issuer
    // The whole warp goes through the waits and one elected lane issues, so that the instructions' operands are uniform
    // for the compiler: with a single lane in the loop a stage took 512 cycles of issuing alone, whatever the tile.
    if (rank == 0) {
      const uint32_t idesc = (I8 ? (2u << 4) | (1u << 7) | (1u << 10) : 1u << 4) | (static_cast<uint32_t>(wa.tile_tok >> 3) << 17) | ((PAIR ? 16u : 8u) << 24);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      const auto wait_all = [&](uint64_t* bar, uint32_t parity) {
        return __all_sync(0xffffffffu, mbar_wait(bar, parity));
      };
      WorkList work = work0;
      Segment sg;
      [[maybe_unused]] long long tr_acc = 0, tr_ab = 0;
      [[maybe_unused]] const long long tr_start = MLD_PAIR_CLOCK();
      for (int nth = 0; ok && work.next(sg); ++nth) {
        const int acc = PAIR ? 0 : nth & 1;
        const uint32_t acc_phase = static_cast<uint32_t>(PAIR ? nth : nth >> 1) & 1u;
        const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(acc * kWtAccCols);
        [[maybe_unused]] const long long t0 = MLD_PAIR_CLOCK();
        if (!wait_all(&tmem_empty[acc], acc_phase ^ 1)) {
          if (lane == 0) atomicExch(a.error, kErrWtBase + 2);
          break;
        }
        tr_acc += MLD_PAIR_CLOCK() - t0;
        tc_after();
        for (int kb = sg.kb0; kb < sg.kb1; ++kb) {
          [[maybe_unused]] const long long t1 = MLD_PAIR_CLOCK();
          if (!wait_all(&full_ab[stage], phase)) {
            if (lane == 0) atomicExch(a.error, kErrWtBase + 3);
            ok = false;
            break;
          }
          tr_ab += MLD_PAIR_CLOCK() - t1;
          tc_after();
          const uint64_t db = make_desc(smem_u32(sX + (size_t)stage * kWtTokBytes));
          const uint32_t ta = tmem_base + kWtACol + static_cast<uint32_t>(stage * 32);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_ts<PAIR, I8>(tmem_d, ta + 8u * k, db + static_cast<uint64_t>((k * 32) >> 4), idesc,
                            (kb > sg.kb0 || k > 0) ? 1u : 0u);
            commit<PAIR>(&empty[stage]);
          }
          __syncwarp();
          if (++stage == kWtStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok && elect_one()) commit<PAIR>(accumulators_ready(sg, work.done(), nth));
        __syncwarp();
      }
#ifdef MLD_TRACE
      if (wa.trace != nullptr && lane == 0) {
        wa.trace[blockIdx.x * 8 + 2] = tr_acc;
        wa.trace[blockIdx.x * 8 + 3] = tr_ab;
        wa.trace[blockIdx.x * 8 + 4] = MLD_PAIR_CLOCK() - tr_start;
      }
#endif
    }
  } else if (warp < 6) {
    // --------------------------------------------------------------------- epilogue
    WorkList work = work0;
    Segment sg;
    int shared = 0;  // segments read by all so far
    for (int nth = 0; work.next(sg); ++nth) {
      const int acc = PAIR ? 0 : nth & 1;
      const bool all = read_by_all(sg, work.done());
      const int use = all ? shared++ : PAIR ? nth : nth >> 1;
      if (!mbar_wait(accumulators_ready(sg, work.done(), nth), static_cast<uint32_t>(use) & 1u)) {
        atomicExch(a.error, kErrWtBase + 4);
        break;
      }
      tc_after();
      if (!drain(sg, 0, all ? kDrainParts : 1, acc)) break;
    }
    if (a.outs.world > 1) __threadfence_system();  // the peer stores are performed before the kernel ends
  } else if (warp == 22) {
    // ------------------------------------------------- producer of the packed weight boxes
    if (lane == 0) prefetch_tmap(&tmap_w);
    int ws = 0;
    uint32_t wphase = 0;
    bool ok = true;
    WorkList work = work0;
    Segment sg;
    while (ok && work.next(sg)) {
      const int nb0 = (tile_n0(sg.tile) + static_cast<int>(rank) * kWtRows) / 4 * BLK;  // byte column of the box
      for (int kb = sg.kb0; kb < sg.kb1; ++kb) {
        if (!__all_sync(0xffffffffu, mbar_wait(&w_empty[ws], wphase ^ 1))) {
          if (lane == 0) atomicExch(a.error, kErrWtBase + 7);
          ok = false;
          break;
        }
        if (elect_one()) {
          mbar_arrive_expect_tx(&full_w[ws], static_cast<uint32_t>(w_stage));
          tma_load_2d(sW + (size_t)ws * w_stage, &tmap_w, &full_w[ws], nb0 / 4, kb * SLICES);  // 32-bit elements
        }
        __syncwarp();
        if (++ws == a.w_stages) {
          ws = 0;
          wphase ^= 1;
        }
      }
    }
  } else {
    // -------------------------------------------------------------------- transform
    const int group = (warp - 6) >> 2;            // this group of four warps takes every fourth stage
    const int quad = warp & 3;                     // the TMEM lane quarter this warp can address
    const int row = quad * 32 + lane;              // output channel of the CTA's 128 = TMEM lane
    const int col4 = row & 3;                      // column of the row inside its 4x4 blocks
    const uint32_t sel8 = static_cast<uint32_t>(col4) | (static_cast<uint32_t>(4 + col4) << 8);
    const __half2 offset = __float2half2_rn(MODE == kModeInt4F16 ? 1032.0f : 1152.0f);  // 1024 + the value of a zero
    [[maybe_unused]] const TurnSelectors turn(col4);
    const int w_shift = __ffs(a.w_stages) - 1;
    bool ok = true;
    int xf_iter = 0;  // stages before the segment
    // A stage's stores are waited for and announced when the next stage's box has been asked for, so that the two trips
    // overlap.
    int stored = -1;
    const auto announce = [&]() {
      if (stored < 0) return;
      tmem_st_wait();
      tc_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR)
          arrive_in_pair(full_ab_lead + stored * 8);
        else
          mbar_arrive(&full_ab[stored]);
      }
      stored = -1;
    };
    WorkList work = work0;
    Segment sg;
    [[maybe_unused]] long long tr_wait = 0, tr_work = 0, tr_st = 0;
    [[maybe_unused]] const long long tr_start = MLD_PAIR_CLOCK();
    int shared = 0;  // segments read by all so far
    for (int nth = 0; ok && work.next(sg); ++nth) {
      const int n = tile_n0(sg.tile) + static_cast<int>(rank) * kWtRows + row;
      const bool scaled = !I8 && n < a.N4 && a.scale != nullptr, blocks = a.scale_mode == MLD_SCALE_BLOCK;
      // 32 input channels are one scale group whenever groups are whole multiples of 32 inputs, the usual case: two loads
      // a stage then, issued when the group's stage before is begun
      const bool one_group = !blocks || (a.group_slices & 7) == 0;
      const __half fixed_scale = __float2half_rn(n < a.N4 ? a.scalar_scale : 0.0f);
      const auto scale_ptr = [&](int slice) {
        int g = !blocks ? 0 : (a.gs_shift >= 0 ? slice >> a.gs_shift : slice / a.group_slices);
        if (g >= a.G) g = a.G - 1;
        return a.scale + (size_t)g * a.N4 + n;
      };
      const auto scale_at = [&](int slice) -> __half { return scaled ? __ldg(scale_ptr(slice)) : fixed_scale; };
      // Asked for a stage of the group ahead, four stages in all, which is more than a trip to HBM.  (The load by hand: it
      // leaves the register alone where there is nothing to load, so that nothing looks at the value, and waits, before the
      // stage that needs it.)
      const auto ask_scale = [&](unsigned short& v, int slice) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.global.nc.u16 %0, [%1];\n\t}"
                     : "+h"(v)
                     : "l"(scale_ptr(slice)), "r"(scaled ? 1u : 0u));
      };
      int kb = sg.kb0 + ((group - xf_iter) & 3);
      unsigned short next0 = __half_as_ushort(fixed_scale), next1 = next0;
      if (kb < sg.kb1) {
        ask_scale(next0, kb * SLICES);
        ask_scale(next1, kb * SLICES + 8);
      }
      for (; kb < sg.kb1; kb += 4) {
        const int iter = xf_iter + kb - sg.kb0, stage = iter & (kWtStages - 1), ws = iter & (a.w_stages - 1);
        const unsigned short cur0 = next0, cur1 = next1;
        if (kb + 4 < sg.kb1) {
          ask_scale(next0, (kb + 4) * SLICES);
          ask_scale(next1, (kb + 4) * SLICES + 8);
        }
        // the packed box has landed (and, below, the stage's tensor-memory columns are free again: their MMAs completed)
        [[maybe_unused]] const long long t0 = MLD_PAIR_CLOCK();
        if (!mbar_wait(&full_w[ws], static_cast<uint32_t>(iter >> w_shift) & 1u)) {
          atomicExch(a.error, kErrWtBase + 5);
          ok = false;
          break;
        }
        [[maybe_unused]] const long long t1 = MLD_PAIR_CLOCK();
        tr_wait += t1 - t0;
        const uint8_t* wp = sW + (size_t)ws * w_stage + (row >> 2) * BLK;
        const uint32_t columns = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + kWtACol + static_cast<uint32_t>(stage * 32);
        if constexpr (I8) {
          const uint32_t* ww = reinterpret_cast<const uint32_t*>(sW + (size_t)ws * w_stage) + row;  // input channel `col4` of the block
          uint32_t in[16];
#pragma unroll
          for (int half = 0; half < 2; ++half) {
#pragma unroll
            for (int i = 0; i < 16; ++i) in[i] = ww[(16 * half + i) * (w_pitch / 4)];
            if (half == 0) {
              announce();
              if (!mbar_wait(&empty[stage], (static_cast<uint32_t>(iter / kWtStages) & 1u) ^ 1u)) {
                atomicExch(a.error, kErrWtBase + 5);
                ok = false;
                break;
              }
              tc_after();
            }
            uint32_t o[16];
#pragma unroll
            for (int i = 0; i < 16; i += 2) turn_blocks(in[i], in[i + 1], turn, o[i], o[i + 1]);
            tmem_st16(columns + static_cast<uint32_t>(16 * half), o);
          }
        } else {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          using Block = typename std::conditional<MODE == kModeInt4F16, uint2, uint4>::type;
          Block blk[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) blk[i] = *reinterpret_cast<const Block*>(wp + (size_t)(8 * half + i) * w_pitch);
          if (half == 0) {
            announce();
            if (!mbar_wait(&empty[stage], (static_cast<uint32_t>(iter / kWtStages) & 1u) ^ 1u)) {
              atomicExch(a.error, kErrWtBase + 5);
              ok = false;
              break;
            }
            tc_after();
          }
          uint32_t o[16];  // o[j] = input channels 32 half + 2j, 2j + 1 of the stage
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const __half2 s2 = __half2half2(one_group ? __ushort_as_half(half == 0 ? cur0 : cur1) : scale_at(kb * SLICES + 2 * (4 * half + c)));
#pragma unroll
            for (int qq = 0; qq < 2; ++qq) {
              const Block v = blk[2 * c + qq];
              if constexpr (MODE == kModeInt4F16) {
                // nibble (k % 4) * 4 + col4: k0, k1 in the halves of .x, k2, k3 in those of .y
                o[4 * c + 2 * qq] = dq_once(((v.x >> (4 * col4)) & 0x000F000Fu) | 0x64006400u, offset, s2);
                o[4 * c + 2 * qq + 1] = dq_once(((v.y >> (4 * col4)) & 0x000F000Fu) | 0x64006400u, offset, s2);
              } else {
                o[4 * c + 2 * qq] = dq_once((__byte_perm(v.x, v.y, sel8) & 0x00FF00FFu) | 0x64006400u, offset, s2);
                o[4 * c + 2 * qq + 1] = dq_once((__byte_perm(v.z, v.w, sel8) & 0x00FF00FFu) | 0x64006400u, offset, s2);
              }
            }
          }
          tmem_st16(columns + static_cast<uint32_t>(16 * half), o);
        }
        }
        if (!ok) break;
        [[maybe_unused]] const long long t2 = MLD_PAIR_CLOCK();
        tr_work += t2 - t1;
        __syncwarp();
        if (lane == 0) mbar_arrive(&w_empty[ws]);  // the box may be overwritten
        stored = stage;
      }
      announce();
      xf_iter += sg.kb1 - sg.kb0;
      if (!ok) break;
      if (!read_by_all(sg, work.done())) continue;
      const int acc = PAIR ? 0 : nth & 1;
      if (!mbar_wait(accumulators_ready(sg, work.done(), nth), static_cast<uint32_t>(shared++) & 1u)) {
        atomicExch(a.error, kErrWtBase + 9);
        break;
      }
      tc_after();
      if (!drain(sg, 1 + group, kDrainParts, acc)) break;
    }
#ifdef MLD_TRACE
    if (wa.trace != nullptr && warp == 6 && lane == 0) {
      wa.trace[blockIdx.x * 8 + 5] = tr_wait;
      wa.trace[blockIdx.x * 8 + 6] = MLD_PAIR_CLOCK() - tr_start;
      wa.trace[blockIdx.x * 8 + 7] = tr_work;
      wa.trace[blockIdx.x * 8 + 0] = tr_st;
    }
#endif
  }
  // Tear-down: nobody leaves while the partner may still arrive on this CTA's barriers or the pair's MMAs
  // may still write this CTA's tensor memory.
  tc_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();
  if (*reinterpret_cast<volatile int*>(a.error) != 0) {
    // a wait ran out somewhere: copies may still be in flight towards this CTA's shared memory
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_after();
    tmem_dealloc_all<PAIR>(tmem_base);
  }
}

}  // namespace

// ------------------------------------------------------------------ host side
#ifdef MLD_TRACE
static long long* g_wt_trace = nullptr;
extern "C" __attribute__((visibility("default"))) void mld_debug_set_wt_trace(void* p) {
  g_wt_trace = static_cast<long long*>(p);
}
#endif

WtGeometry wtmem_geometry(int M, int N, int K, int mode, int sms, bool may_share) {
  WtGeometry g;
  const int N4 = align_n(N, 4);
  const bool i8 = mode == kModeInt8I8;
  g.kp = align_n(K, i8 ? 16 : 8);
  g.k_blocks = div_up(g.kp, i8 ? 128 : 64);
  // Up to 128 tokens a CTA works alone; with more, pairs share the fetching of the tokens.
  g.ctas = M <= 128 || sms < 2 ? 1 : 2;
  g.n_tiles = div_up(N4, g.ctas * kWtRows);
  const int most = 128 * g.ctas;
  g.tile_tok = M >= most ? most : align_n(M, i8 && g.ctas == 2 ? 32 : 16);
#ifdef MLD_TRACE
  if (const char* e = getenv("MLD_WT_TOK")) g.tile_tok = atoi(e);
#endif
  g.tok_tiles = div_up(M, g.tile_tok);
  const int pairs = sms < 2 ? 1 : sms / 2 * 2 / g.ctas;  // (the split workspace has a slot per CTA of sms / 2 pairs)
  const long tiles = (long)g.n_tiles * g.tok_tiles;
  // The last whole wave of tiles and the remainder are cut along K and dealt out evenly; so are the tiles of a launch
  // that has fewer of them than pairs (43 tiles of 4096 x 11008 left 31 of 74 pairs without work), into parts of eight
  // stages or more, of an eighth of a tile at least (a tile that does not begin with a part has nine): the pair that
  // completes a tile reads the other parts' accumulators
  // one after another, which costs about as much as a few stages.
  const bool few = tiles < pairs;
  g.shares_tiles = may_share && tiles % pairs != 0;
  if (g.shares_tiles) {
    g.shared_tiles = static_cast<int>(few ? tiles : pairs + tiles % pairs);
    const long units = (long)g.shared_tiles * g.k_blocks;
    g.units_per_pair = static_cast<int>((units + pairs - 1) / pairs);
    int least = div_up(g.k_blocks, 8);
    if (least < 8) least = 8;
    if (least > g.k_blocks) least = g.k_blocks;
    if (g.units_per_pair < least) g.units_per_pair = least;
    g.grid = g.ctas * static_cast<int>(few ? (units + g.units_per_pair - 1) / g.units_per_pair : pairs);
  } else {
    g.shared_tiles = 0;
    g.units_per_pair = 0;
    g.grid = g.ctas * static_cast<int>(few ? tiles : pairs);
  }
  const int blk = mode == kModeInt4F16 ? 8 : 16;
  const int w_stage = (i8 ? 32 : 16) * (kWtRows / 4) * blk;
  const int fixed = 1024 + (2 * 24 + 2 * kWtStages + 5) * 8 + 64;
  int ws = (226 * 1024 - fixed - kWtStages * kWtTokBytes) / w_stage;
  g.w_stages = ws >= 16 ? 16 : ws >= 8 ? 8 : 4;  // (a power of two)
  g.smem_bytes = (size_t)kWtStages * kWtTokBytes + (size_t)ws * w_stage + fixed;
  return g;
}

int launch_gemm_wtmem(int mode, const void* x_kmajor, const void* packed, const WtGeometry& g, int M, int N, int K,
                      const void* scale, int scale_mode, int G, int group_slices, float scalar_scale, const void* bias,
                      const float* a_params, const int32_t* w_sum, void* y, int dst_layout, int* error, cudaStream_t stream,
                      const PeerOutputs* outs, const PairSplit* split) {
  if (mode != kModeInt4F16 && mode != kModeInt8F16 && mode != kModeInt8I8) {
    set_last_error_text("bad GEMM mode");
    return MLD_INVALID_ARGUMENT;
  }
  if (g.shares_tiles && (split == nullptr || split->ws == nullptr || split->flags == nullptr || split->epoch == 0)) {
    set_last_error_text("this GEMM geometry shares tiles between SM pairs and needs a split workspace");
    return MLD_INVALID_ARGUMENT;
  }
  const int N4 = align_n(N, 4);
  const int blk = mode == kModeInt4F16 ? 8 : 16;
  const int SS = div_up(K, 4), DS = N4 / 4;
  const bool i8 = mode == kModeInt8I8;
  CUtensorMap tx, tw;
  // activations: K-major rows [M][kp]; box = one swizzle atom of K x this CTA's half of the tile's tokens
  const int esz = i8 ? 1 : 2;
  int rc = make_tmap_2d(&tx, x_kmajor, (uint64_t)g.kp * esz, M, (uint64_t)g.kp * esz, kKBytes, g.tile_tok / g.ctas, esz,
                        CU_TENSOR_MAP_SWIZZLE_128B, i8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, true);
  if (rc != MLD_OK) return rc;
  // packed weights: [K/4] rows of N4/4 blocks; box = one stage's rows x the CTA's 32 blocks, in 32-bit elements
  rc = make_tmap_2d(&tw, packed, (uint64_t)DS * blk, SS, (uint64_t)DS * blk, (kWtRows / 4) * blk, i8 ? 32 : 16, 4,
                    CU_TENSOR_MAP_SWIZZLE_NONE);
  if (rc != MLD_OK) return rc;
  WtArgs wa;
  memset(&wa, 0, sizeof wa);
  PairArgs& a = wa.p;
  a.M = M;
  a.N = N;
  a.N4 = N4;
  a.m_tiles = g.tok_tiles;  // the work list's "tile % m_tiles" runs over the token tiles
  a.n_tiles = g.n_tiles;
  a.k_blocks = g.k_blocks;
  a.w_stages = g.w_stages;
  a.scale = scale_mode == MLD_SCALE_SCALAR ? nullptr : static_cast<const __half*>(scale);
  a.scale_mode = scale_mode;
  a.G = G;
  a.group_slices = group_slices;
  a.gs_shift = -1;
  for (int sh = 0; sh < 24; ++sh)
    if ((1 << sh) == group_slices) a.gs_shift = sh;
  a.scalar_scale = scalar_scale;
  a.bias = bias;
  a.a_params = a_params;
  a.w_sum = w_sum;
  a.y = y;
  a.dst_layout = dst_layout;
  a.error = error;
  a.shared_tiles = g.shared_tiles;
  a.units_per_pair = g.units_per_pair;
  if (g.shares_tiles) {
    a.split_ws = split->ws;
    a.split_flags = split->flags;
    a.epoch = split->epoch;
  }
  if (outs != nullptr && outs->world > 1 && dst_layout == MLD_LAYOUT_SLICED) a.outs = *outs;
  wa.tile_tok = g.tile_tok;
  wa.tok_tiles = g.tok_tiles;
#ifdef MLD_TRACE
  wa.trace = g_wt_trace;
  wa.trace_flags = getenv("MLD_WT_FLAGS") != nullptr ? atoi(getenv("MLD_WT_FLAGS")) : 0;
#endif
  void (*kern)(CUtensorMap, CUtensorMap, WtArgs) =
      g.ctas == 2 ? (mode == kModeInt4F16   ? gemm_wtmem_kernel<kModeInt4F16, true>
                     : mode == kModeInt8F16 ? gemm_wtmem_kernel<kModeInt8F16, true>
                                            : gemm_wtmem_kernel<kModeInt8I8, true>)
                  : (mode == kModeInt4F16   ? gemm_wtmem_kernel<kModeInt4F16, false>
                     : mode == kModeInt8F16 ? gemm_wtmem_kernel<kModeInt8F16, false>
                                            : gemm_wtmem_kernel<kModeInt8I8, false>);
  static bool configured[2][3][kMaxDevices];
  bool(&done)[kMaxDevices] = configured[g.ctas - 1][mode];
  int dev;
  if (needs_configure(done, &dev)) {
    MLD_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    if (dev >= 0) done[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.grid, 1, 1);
  cfg.blockDim = dim3(kWtThreads, 1, 1);
  cfg.dynamicSmemBytes = g.smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g.ctas == 2 ? 2 : 1;
  MLD_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, tx, tw, wa));
  count_launch();
  return MLD_OK;
}

}  // namespace mld
