// Small-m ("decode-shaped") MX GEMM for sm_100a: D (m x n, m <= 64) = A (m x k) * B (n x k)^T
// with OCP MX fp8 / fp4 operands and one E8M0 scale per 32 k-elements.  The CPU library has
// no kernel of its own for this shape (its GEMV-like calls run the general blocked path,
// gemm/kernel/run_blocked.h:79-174, and spend their time decoding B,
// gemm/threadblock/mma_policy_mx.h:171-257).  On the GPU the shape is bound by reading the
// weight matrix B once from HBM, so everything here serves one goal: start that stream
// early, keep every SM pulling on it, and add no second launch.
//
// Kernel view: the weights W (the caller's B, `Mk` rows of k) sit on the MMA M side in
// 128-row tiles, the activations X (the caller's A, `Nk` <= BN rows) on the N side.
//
//   * One launch.  Four warps (thread = tile row) fetch the raw row-major scale bytes
//     themselves, 16 bytes per row at a time and a few fetches ahead (cp.async into a small
//     staging ring), and turn them into the 512-byte atoms that tcgen05.cp wants, in shared
//     memory, ahead of the MMAs.  (Measured: a 16-byte wide TMA box per stage instead costs
//     the TMA unit as much time as the 128-byte wide operand box -- it works row by row --
//     and halved the stream.)
//   * A CTA takes whole tiles while there are enough of them to fill the SMs.  When there are
//     fewer, a cluster of 2 to 6 CTAs shares each tile, every CTA a contiguous part of k: the
//     partial accumulators meet in distributed shared memory (st.async straight into the
//     owner's buffer, its barrier counting the bytes), and each owner adds the pieces of its
//     part in ascending k order - a fixed order, so results do not depend on which CTA
//     finished first.  The cut of a tile never leaves the chip and needs no workspace.
//   * A CTA's part of k may be summed in pieces (kPieces).  The tensor cores drop the low bits of a running
//     sum: against float64, 8-bit results are off by 6e-10 per element of k summed in one
//     accumulator.  Where few tiles leave every CTA a long part, the two accumulators take turns every
//     p.piece_kb k-blocks and the epilogue warps add them up in f32, in ascending k order, in tensor
//     memory beside them, while the MMAs of the next piece run.  m = 32, 1024 weight rows x k =
//     14336, e4m3: 1.4e-6 off in one sum of 19 k-blocks, 4.1e-7 in pieces of 5; 9.3 us / 9.6.
//   * Launched with programmatic stream serialization: a CTA may become resident and set up
//     its barriers and tensor memory while the kernel before this one in the stream is
//     still finishing; every role then waits (griddepcontrol.wait) before it reads or
//     writes global memory.
//
// Where the time of one call goes (14336 x 4096 fp4 weights, m = 1, calls back to back over
// weights that are not in L2: 8.4 us per call; time stamps of every role in an instrumented
// build): the HBM stream itself 5.0 us (5.9 TB/s), the latency of the first bytes after the
// wait 1.3 us, the tail after the last byte and the gap between a kernel's last CTA leaving
// and its successor passing the wait 1 us each.  Cutting a tile's k over a cluster instead of
// through partial sums in global memory (a chain of dependent L2 round trips of about 4 us):
// e4m3 m = 32, 4096 weight rows x k = 14336 21.2 -> 14.4 us, x k = 4096 15.5 -> 8.9 us;
// e2m1 m = 1, 4096 x 14336 16.1 -> 9.8 us; 1024 x 4096 8.7 -> 5.1 us.
//
// Tried and not kept, each measured on the same loop: asking W into L2 ahead of the wait,
// with untiled bulk prefetches of the CTA's whole share (8.4 -> 10.3 us: they queue in the
// same unit as the loads), with prefetch instructions for the first 2, 4, 8 or 12 k-blocks
// (within 0.3 us either way), with 256-byte fill hints or TMA prefetch boxes; two smaller
// CTAs per SM so that the next call's CTAs sit beside this call's (8.4 -> 9.3 us: the
// shallower ring slows the stream by what the overlap saves), with and without prefetch.
//
// Roles (320 threads): warp 0 TMA producer, warp 1 MMA issuer (owns tensor memory), warps
// 2-5 scale writers (thread = tile row), warps 6-9 epilogue (one TMEM lane quarter each).
// A stage's "full" barrier collects the TMA bytes and the four writer warps' arrivals, so
// the MMA warp waits once per stage; the writers handle the units of one 16-byte scale
// fetch together (one proxy fence per fetch, not per unit).
// Every wait is bounded, as in the general kernel.
#pragma once

#include "epilogue.cuh"
#include "gemm_params.h"
#include "ptx_sm100.cuh"
#include "ptx_sm100_pair.cuh"

namespace b200 {

constexpr int kDecodeThreads = 320;
constexpr int kDecodeSfSlots = 4;    // tensor-memory scale slots the MMA warp rotates over
constexpr int kDecodeMaxStages = 12;
constexpr int kDecodeFetchAhead = 4; // 16-byte scale chunks each writer thread keeps in flight

struct DecodeParams {
  int32_t Mk, Nk;            // rows of W (caller's n), rows of X (caller's m, <= BN)
  int32_t kblocks32;         // valid scale bytes per row, ceil(k / 32)
  int32_t ld_sw, ld_sx;      // leading dimensions of the two scale arrays (bytes)
  const uint8_t* sw;         // W's scales (row-major, 16-byte aligned rows)
  const uint8_t* sx;         // X's scales
  int32_t tiles, k_blocks;   // 128-row tiles of W, 128-byte k-blocks
  int32_t BN;                // 32 or 64
  int32_t stages;
  int32_t splits;            // CTAs (one cluster) that share a tile's k; 1: whole tiles per CTA
  int32_t piece_kb;          // kPieces: k-blocks summed in one accumulator
  int32_t tmem_cols;         // power of two >= 2 (kPieces: 3) * BN + kDecodeSfSlots * scale columns per unit
  uint32_t idesc;
  uint32_t wait_budget_us;   // budget of every bounded wait
  EpilogueParams epi;
  int32_t* error;
#ifdef CPUOPS_B200_INSTRUMENT
  unsigned long long* clk;   // instrumented build: min / max over CTAs of role time stamps (ns)
#endif
};

// Instrumented build: time stamp `slot` of this launch (even word: the earliest CTA, kept as
// the maximum of ~t so that an all-zero buffer means "nothing yet"; odd word: the latest).
#ifdef CPUOPS_B200_INSTRUMENT
#define DECODE_STAMP(p, slot, lane_ok)                                                    \
  do {                                                                                    \
    if ((p).clk != nullptr && (lane_ok)) {                                                \
      const unsigned long long t__ = global_timer_ns();                                   \
      atomicMax((p).clk + 2 * (slot), ~t__);                                              \
      atomicMax((p).clk + 2 * (slot) + 1, t__);                                           \
    }                                                                                     \
  } while (0)
#else
#define DECODE_STAMP(p, slot, lane_ok) do { } while (0)
#endif

// Shared-memory footprint: per stage the W tile, the X tile (its Nk rows, rounded up so that
// the next stage stays 1024-byte aligned) and the scale atoms of both; then the writers'
// staging ring and the barriers.
__host__ __device__ inline int decode_x_bytes(int Nk) { return (Nk * 128 + 1023) / 1024 * 1024; }
__host__ __device__ inline int decode_stage_bytes(int Nk) { return kTileM * 128 + decode_x_bytes(Nk); }
__host__ __device__ inline int decode_staging_bytes(int BN) { return kDecodeFetchAhead * (kTileM + BN) * 16; }
constexpr int kDecodeBarrierBytes = 512;
// The reduction works in units of one lane quarter (32 rows) x 16 columns: 2 KB per source CTA.
// Unit u belongs to CTA u % splits of the cluster, as its slot u / splits.
constexpr int kDecodeUnitBytes = 32 * 16 * 4;
__host__ __device__ inline int decode_reduce_units(int Nk) { return 4 * ((Nk + 15) / 16); }
__host__ __device__ inline int decode_reduce_bytes(int Nk, int splits) {
  if (splits <= 1) return 0;
  return (decode_reduce_units(Nk) + splits - 1) / splits * splits * kDecodeUnitBytes;
}
constexpr int kDecodeMaxSplits = 6;
constexpr int kDecodeMaxSlots = 8;  // 16 units over at least 2 CTAs
__host__ __device__ inline int decode_smem_bytes(int Nk, int BN, int stages, int atoms_per_unit, int splits) {
  return 1024 + stages * (decode_stage_bytes(Nk) + atoms_per_unit * 512) + decode_staging_bytes(BN) +
         decode_reduce_bytes(Nk, splits) + kDecodeBarrierBytes;
}

// alpha * acc + beta * C, the chain ops, and the store of one N-column chunk of one row.
template <int N>
__device__ __forceinline__ void decode_store_chunk(const EpilogueParams& e, uint32_t (&r)[N], int krow,
                                                   int kcol0, int ncols) {
  uint32_t src[N];
  if (e.beta_nonzero) {
    const uint32_t* c = static_cast<const uint32_t*>(e.C) + (krow * e.c_sr + kcol0 * e.c_sc);
#pragma unroll
    for (int i = 0; i < N; ++i) src[i] = i < ncols ? c[i * e.c_sc] : 0u;
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) src[i] = 0u;
  }
#pragma unroll
  for (int i = 0; i < N; ++i) r[i] = linear_combine_bits<false>(e, r[i], src[i]);
  for (int t = 0; t < e.n_ops; ++t) apply_op_chunk<false, N>(e.ops[t], r, krow, kcol0, ncols);
  uint32_t* d = static_cast<uint32_t*>(e.D) + (krow * e.d_sr + kcol0 * e.d_sc);
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i < ncols) d[i * e.d_sc] = r[i];
}

__device__ __forceinline__ uint32_t pick_word(const uint4& v, int i) {
  return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w));
}

__device__ __forceinline__ uint32_t add_f32(uint32_t a, uint32_t b) {
  return __float_as_uint(__fadd_rn(__uint_as_float(a), __uint_as_float(b)));
}

template <int KIND, bool kPieces>
__global__ void __launch_bounds__(kDecodeThreads, 1)
    decode_mx_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                     const DecodeParams p) {
  static_assert(KIND == kKindMxf8 || KIND == kKindMxf4, "MX kinds only");
  // scale bytes per row per unit: 128 fp8 elements = 4 blocks, 256 fp4 elements = 8
  constexpr int kSfBytes = KIND == kKindMxf4 ? 8 : 4;
  constexpr int kKa = kSfBytes / 4;           // atoms along k per operand per unit
  constexpr int kUnitsPerChunk = 16 / kSfBytes;  // units served by one 16-byte fetch of a scale row
  constexpr uint32_t kSfCols = 4u * 2u * kKa; // tensor-memory columns of one unit's scales
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  DECODE_STAMP(p, 0, threadIdx.x == 0);

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t pad = ((raw_addr + 1023u) & ~1023u) - raw_addr;
  uint8_t* smem = smem_raw + pad;
  const uint32_t smem_base = raw_addr + pad;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int stages = p.stages, BN = p.BN;
  const uint32_t stage_bytes = static_cast<uint32_t>(decode_stage_bytes(p.Nk));
  const uint32_t atom_bytes = 2u * kKa * 512u;
  const uint32_t atom_base = smem_base + stages * stage_bytes;
  const uint32_t staging_base = atom_base + stages * atom_bytes;
  const uint32_t red_base = staging_base + static_cast<uint32_t>(decode_staging_bytes(BN));
  const uint32_t bar_base = red_base + static_cast<uint32_t>(decode_reduce_bytes(p.Nk, p.splits));
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kDecodeMaxStages + s); };
  auto acc_full_bar = [&](int b) { return bar_base + 8u * (2 * kDecodeMaxStages + b); };
  auto acc_empty_bar = [&](int b) { return bar_base + 8u * (2 * kDecodeMaxStages + 2 + b); };
  const uint32_t drain_bar = bar_base + 8u * (2 * kDecodeMaxStages + 4);
  auto red_bar = [&](int slot) { return bar_base + 8u * (2 * kDecodeMaxStages + 5 + slot); };
  constexpr int kBarriers = 2 * kDecodeMaxStages + 5 + kDecodeMaxSlots;
  static_assert(8 * kBarriers + 8 <= kDecodeBarrierBytes, "barrier region too small");
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + (bar_base - smem_base) + 8 * kBarriers);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint64_t budget_ns = static_cast<uint64_t>(p.wait_budget_us) * 1000ull;

  // This CTA's units: its cluster's tiles x its part of k.
  const int splits = p.splits;
  const int rank = splits > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
  const int groups = static_cast<int>(gridDim.x) / splits, group = static_cast<int>(blockIdx.x) / splits;
  const int tile0 = static_cast<int>(static_cast<int64_t>(group) * p.tiles / groups);
  const int tile1 = static_cast<int>(static_cast<int64_t>(group + 1) * p.tiles / groups);
  const int kb0 = static_cast<int>(static_cast<int64_t>(rank) * p.k_blocks / splits);
  const int kb1 = static_cast<int>(static_cast<int64_t>(rank + 1) * p.k_blocks / splits);
  const int n_units = (tile1 - tile0) * (kb1 - kb0);

  if (warp == 2) {
    for (int i = lane; i < kBarriers; i += 32) {
      // full: the producer's arrive.expect_tx plus one arrival per scale-writer warp (the
      // phase completes when the operand tiles have landed AND the stage's atoms are
      // written: one wait for the MMA warp); empty / accumulator full / drain: one
      // tcgen05.commit; accumulator empty: one arrival per epilogue warp
      uint32_t count = 1u;
      if (i < kDecodeMaxStages) count = 5u;
      if (i == 2 * kDecodeMaxStages + 2 || i == 2 * kDecodeMaxStages + 3) count = 4u;
      mbar_init(bar_base + 8u * static_cast<uint32_t>(i), count);
    }
    if (lane == 0) *abort_flag = 0;
    fence_mbar_init();
    __syncwarp();
    // reduction slots: all pieces of this CTA's units, in bytes
    if (splits > 1 && lane < kDecodeMaxSlots && rank + lane * splits < decode_reduce_units(p.Nk))
      mbar_expect_tx(red_bar(lane), static_cast<uint32_t>(splits * kDecodeUnitBytes));
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), static_cast<uint32_t>(p.tmem_cols));
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmW);
    prefetch_tensormap(&tmX);
  }
  tc_fence_before_sync();
  // (the epilogue warps wait for this arrival of every CTA of the cluster before they send
  // anything: the reduction barriers are armed by then)
  if (splits > 1) cluster_arrive();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  DECODE_STAMP(p, 1, threadIdx.x == 0);

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    // The whole warp runs the loop, one elected lane issues.  Per unit: the W tile (128
    // rows x 128 bytes of k) and the X tile (exactly its Nk rows: a box with rows outside
    // the tensor costs the TMA unit time for every such row).
    const uint32_t el = elect_one() ? 1u : 0u;
    const uint32_t tx_bytes = static_cast<uint32_t>(kTileM * 128 + p.Nk * 128);
    auto issue_w = [&](int s, int tile, int kb) {
      tma_load_2d_g<false>(smem_base + s * stage_bytes, &tmW, full_bar(s), kb * 128, tile * kTileM, el);
    };
    auto issue_x = [&](int s, int kb) {
      tma_load_2d_g<false>(smem_base + s * stage_bytes + kTileM * 128, &tmX, full_bar(s), kb * 128, 0, el);
    };
    asm volatile("griddepcontrol.wait;" ::: "memory");
    DECODE_STAMP(p, 2, el);
    int s = 0, tile = tile0, kb = kb0;
    uint32_t ph = 0;
    for (int i = 0; i < n_units; ++i) {
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(empty_bar(s), ph ^ 1u, abort_flag, budget_ns))) {
        if (el) {
          leave_error(p.error, kErrProducerWait);
          *abort_flag = 1;
        }
        break;
      }
      mbar_expect_tx_p(full_bar(s), tx_bytes, el);
      issue_w(s, tile, kb);
      issue_x(s, kb);
      if (++kb == kb1) { kb = kb0; ++tile; }
      if (++s == stages) { s = 0; ph ^= 1u; }
    }
    DECODE_STAMP(p, 3, el);
    if (*abort_flag != 0 && el) {
      // give the copies already issued time to land before the CTA exits
      const uint64_t t_end = global_timer_ns() + 200000;
      while (global_timer_ns() < t_end) __nanosleep(1000);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------- MMA issuer -------------------------------
    const uint32_t el = elect_one() ? 1u : 0u;
    constexpr uint32_t kAll = 0xffffffffu;
    const uint64_t op_hi64 = make_smem_desc_hi(16, 1024, 2);  // K-major, 128-byte swizzle
    const uint32_t op_hi = static_cast<uint32_t>(op_hi64 >> 32);
    const uint32_t a_lo0 = static_cast<uint32_t>(op_hi64) | (smem_base >> 4);
    const uint32_t b_lo0 = static_cast<uint32_t>(op_hi64) | ((smem_base + kTileM * 128) >> 4);
    const uint64_t sf_hi64 = make_smem_desc_hi(0, 128, 0);
    const uint32_t sf_hi = static_cast<uint32_t>(sf_hi64 >> 32);
    const uint32_t sf_lo0 = static_cast<uint32_t>(sf_hi64) | (atom_base >> 4);
    const uint32_t idesc = p.idesc;
    uint32_t id1 = idesc, id2 = idesc, id3 = idesc;
    if constexpr (KIND == kKindMxf8) {
      id1 = idesc_with_sf_ids(idesc, 1, 1);
      id2 = idesc_with_sf_ids(idesc, 2, 2);
      id3 = idesc_with_sf_ids(idesc, 3, 3);
    } else {
      id1 = idesc_with_sf_ids(idesc, 2, 2);
      id3 = id1;
    }
    const uint32_t sf_t0 = tmem_base + 2u * static_cast<uint32_t>(BN);
    int s = 0, buf = 0, sf_q = 0;
    uint32_t ph = 0, acc_ph = 0;
    bool ok = true;
    int i = 0;
    [[maybe_unused]] int tile_left = kb1 - kb0;
    while (i < n_units && ok) {
      const int piece_units = kPieces ? min(tile_left, p.piece_kb) : kb1 - kb0;  // ... or one tile
      if (!__all_sync(kAll, mbar_wait_bounded(acc_empty_bar(buf), acc_ph ^ 1u, abort_flag, budget_ns))) {
        if (el) {
          leave_error(p.error, kErrMmaWaitAcc);
          *abort_flag = 1;
        }
        ok = false;
        break;
      }
      tc_fence_after_sync();
      const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf * BN);
      uint32_t accumulate = 0;
      for (int j = 0; j < piece_units; ++j) {
        // the stage's operand tiles have landed and its scale atoms are written
        if (!__all_sync(kAll, mbar_wait_bounded(full_bar(s), ph, abort_flag, budget_ns))) {
          if (el) {
            leave_error(p.error, kErrMmaWaitFull);
            *abort_flag = 1;
          }
          ok = false;
          break;
        }
        tc_fence_after_sync();
        if (i == 0 && j == 0) DECODE_STAMP(p, 4, el);
        if (i + j + 1 == n_units) DECODE_STAMP(p, 5, el);
        const uint32_t a_lo = a_lo0 + s * (stage_bytes >> 4), b_lo = b_lo0 + s * (stage_bytes >> 4);
        const uint32_t sfa_t = sf_t0 + static_cast<uint32_t>(sf_q) * kSfCols, sfb_t = sfa_t + 4u * kKa;
        {
          uint32_t src = sf_lo0 + s * (atom_bytes >> 4), dst = sfa_t;
          for (uint32_t a = 0; a < 2u * kKa; ++a, src += 32, dst += 4) tmem_cp_atom_g<false>(dst, src, sf_hi, el);
        }
        if constexpr (KIND == kKindMxf8) {
          mma_mxf8f6f4_g<false>(d_tmem, a_lo, op_hi, b_lo, op_hi, idesc, sfa_t, sfb_t, accumulate, el);
          mma_mxf8f6f4_g<false>(d_tmem, a_lo + 2, op_hi, b_lo + 2, op_hi, id1, sfa_t, sfb_t, 1u, el);
          mma_mxf8f6f4_g<false>(d_tmem, a_lo + 4, op_hi, b_lo + 4, op_hi, id2, sfa_t, sfb_t, 1u, el);
          mma_mxf8f6f4_g<false>(d_tmem, a_lo + 6, op_hi, b_lo + 6, op_hi, id3, sfa_t, sfb_t, 1u, el);
        } else {
          mma_mxf4_g<false>(d_tmem, a_lo, op_hi, b_lo, op_hi, idesc, sfa_t, sfb_t, accumulate, el);
          mma_mxf4_g<false>(d_tmem, a_lo + 2, op_hi, b_lo + 2, op_hi, id1, sfa_t, sfb_t, 1u, el);
          mma_mxf4_g<false>(d_tmem, a_lo + 4, op_hi, b_lo + 4, op_hi, id2, sfa_t + 4u, sfb_t + 4u, 1u, el);
          mma_mxf4_g<false>(d_tmem, a_lo + 6, op_hi, b_lo + 6, op_hi, id3, sfa_t + 4u, sfb_t + 4u, 1u, el);
        }
        accumulate = 1u;
        tc_commit_g<false>(empty_bar(s), el);  // frees the stage once these MMAs and copies have read it
        if (++sf_q == kDecodeSfSlots) sf_q = 0;
        if (++s == stages) { s = 0; ph ^= 1u; }
      }
      if (!ok) break;
      tc_commit_g<false>(acc_full_bar(buf), el);
      if (++buf == 2) { buf = 0; acc_ph ^= 1u; }
      i += piece_units;
      if constexpr (kPieces) {
        tile_left -= piece_units;
        if (tile_left == 0) tile_left = kb1 - kb0;
      }
    }
    // nothing may still be executing when tensor memory is released
    tc_commit_g<false>(drain_bar, el);
    int dummy = 0;
    if (!__all_sync(kAll, mbar_wait_bounded(drain_bar, 0, &dummy, budget_ns)) && el) {
      leave_error(p.error, kErrDrainWait);
      *abort_flag = 1;
    }
    __syncwarp();
  } else if (warp < 6) {
    // ------------------------------ scale writers ------------------------------
    // Thread r (0..127) owns row r of the W tile and, if r < Nk, row r of X.  It fetches its
    // rows' scale bytes 16 at a time (one chunk = 2 fp4 units or 4 fp8 units) into its own
    // 16-byte slots of a staging ring, kDecodeFetchAhead chunks ahead, and reads them back
    // itself (cp.async.wait_group orders a thread's own copies: no barrier needed).  For
    // every unit it then writes one word per atom at byte (r % 32) * 16 + (r / 32) * 4.
    // Bytes past ceil(k/32) and rows past the matrix are never read (they are zero-filled:
    // the finite scale 2^-127 against all-zero data); X rows that do not exist get 0x7F.
    const int r = (warp - 2) * 32 + lane;
    const uint32_t slot_off = static_cast<uint32_t>((r & 31) * 16 + (r >> 5) * 4);
    const uint32_t stage_w = staging_base + static_cast<uint32_t>(r) * 16u;
    const uint32_t stage_x = stage_w + kTileM * 16u;
    const uint32_t kStagingSlot = static_cast<uint32_t>(kTileM + BN) * 16u;
    const bool has_x = r < p.Nk;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int f_i = 0, f_tile = tile0, f_kb = kb0;  // fetch cursor: the next chunk starts at this unit
    auto fetch = [&](int slot) {
      if (f_i < n_units) {
        const int col = (f_kb * kSfBytes) >> 4;
        const int row = f_tile * kTileM + r;
        const int valid_w = row < p.Mk ? min(16, p.kblocks32 - col * 16) : 0;
        const uint8_t* src_w = p.sw + static_cast<int64_t>(min(row, p.Mk - 1)) * p.ld_sw + col * 16;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(stage_w + slot * kStagingSlot),
                     "l"(src_w), "r"(valid_w)
                     : "memory");
        if (has_x) {
          const uint8_t* src_x = p.sx + static_cast<int64_t>(r) * p.ld_sx + col * 16;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(stage_x + slot * kStagingSlot),
                       "l"(src_x), "r"(min(16, p.kblocks32 - col * 16))
                       : "memory");
        }
        const int next_kb = (f_kb | (kUnitsPerChunk - 1)) + 1;
        if (next_kb >= kb1) {
          f_i += kb1 - f_kb;
          f_kb = kb0;
          ++f_tile;
        } else {
          f_i += next_kb - f_kb;
          f_kb = next_kb;
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");  // always: the group count stays in step
    };
    for (int j = 0; j < kDecodeFetchAhead; ++j) fetch(j);
    int s = 0, kb = kb0, c_slot = 0, i = 0;
    uint32_t ph = 0;
    uint4 cur_w = make_uint4(0, 0, 0, 0), cur_x = make_uint4(0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
    bool alive = true;
    while (i < n_units && alive) {
      // one chunk: the units that share this 16-byte fetch (up to the end of this CTA's part of k)
      const int in_chunk = min(kUnitsPerChunk - (kb & (kUnitsPerChunk - 1)), kb1 - kb);
      asm volatile("cp.async.wait_group %0;" ::"n"(kDecodeFetchAhead - 1) : "memory");
      asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(cur_w.x), "=r"(cur_w.y), "=r"(cur_w.z), "=r"(cur_w.w)
                   : "r"(stage_w + c_slot * kStagingSlot));
      if (has_x)
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(cur_x.x), "=r"(cur_x.y), "=r"(cur_x.z), "=r"(cur_x.w)
                     : "r"(stage_x + c_slot * kStagingSlot));
      int s2 = s;
      uint32_t ph2 = ph;
      for (int u = 0; u < in_chunk; ++u) {
        // the stage's previous atoms have been copied to tensor memory (its MMAs are done)
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(empty_bar(s2), ph2 ^ 1u, abort_flag, budget_ns))) {
          if (lane == 0) {
            leave_error(p.error, kErrProducerWait);
            *abort_flag = 1;
          }
          alive = false;
          break;
        }
        const int sub = ((kb + u) & (kUnitsPerChunk - 1)) * kKa;  // first word of this unit within the chunk
        const uint32_t aw = atom_base + s2 * atom_bytes + slot_off, ax = aw + kKa * 512u;
#pragma unroll
        for (int a = 0; a < kKa; ++a) {
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(aw + 512u * a), "r"(pick_word(cur_w, sub + a)) : "memory");
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(ax + 512u * a), "r"(pick_word(cur_x, sub + a)) : "memory");
        }
        if (++s2 == stages) { s2 = 0; ph2 ^= 1u; }
      }
      if (!alive) break;
      fence_proxy_async_shared_cta();  // these writes -> visible to tcgen05.cp (one fence per chunk)
      __syncwarp();
      if (lane == 0) {
        int s3 = s;
        for (int u = 0; u < in_chunk; ++u) {
          mbar_arrive(full_bar(s3));
          if (++s3 == stages) s3 = 0;
        }
      }
      // the chunk is in registers (the stores above used it): its slot takes the next fetch
      fetch(c_slot);
      if (++c_slot == kDecodeFetchAhead) c_slot = 0;
      s = s2;
      ph = ph2;
      i += in_chunk;
      kb += in_chunk;
      if (kb == kb1) kb = kb0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  } else {
    // -------------------------------- epilogue --------------------------------
    asm volatile("griddepcontrol.wait;" ::: "memory");  // before C is read, D written
    const int q = warp & 3;  // the TMEM lane quarter this warp can read
    const int nchunks = (p.Nk + 15) / 16;
    const EpilogueParams& e = p.epi;
    warm_epilogue_params(e);
    int buf = 0;
    uint32_t acc_ph = 0;
    bool alive = true;
    if (splits > 1) cluster_wait();
    // kPieces: the sum of a tile's finished pieces, behind the accumulators and the scale slots
    const uint32_t tsum =
        tmem_base + (static_cast<uint32_t>(q * 32) << 16) + 2u * static_cast<uint32_t>(BN) + kDecodeSfSlots * kSfCols;
    for (int tile = tile0; tile < tile1; ++tile) {
      // the accumulator is in registers: hand the buffer back to the MMA warp
      auto hand_back = [&]() {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty_bar(buf));
      };
      [[maybe_unused]] bool summed = false;
      if constexpr (kPieces) {  // all pieces of this CTA's part of k but the last
        for (int left = kb1 - kb0; left > p.piece_kb && alive; left -= p.piece_kb) {
          const bool ready = mbar_wait_bounded(acc_full_bar(buf), acc_ph, abort_flag, budget_ns);
          if (!__all_sync(0xffffffffu, ready)) {
            alive = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t from = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(buf * BN);
#pragma unroll 1
          for (int c = 0; c < p.Nk; c += 16) {
            uint32_t v[16], w[16];
            tmem_ld_32x16(from + static_cast<uint32_t>(c), v);
            if (summed) tmem_ld_32x16(tsum + static_cast<uint32_t>(c), w);
            tmem_ld_wait();
            if (summed) {
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = add_f32(w[j], v[j]);
            }
            tmem_st_32x16(tsum + static_cast<uint32_t>(c), v);
          }
          tmem_st_wait();
          hand_back();
          if (++buf == 2) { buf = 0; acc_ph ^= 1u; }
          summed = true;
        }
      }
      const bool got = alive && mbar_wait_bounded(acc_full_bar(buf), acc_ph, abort_flag, budget_ns);
      if (!__all_sync(0xffffffffu, got)) {
        if (lane == 0) {
          leave_error(p.error, kErrEpilogueWait);
          *abort_flag = 1;
        }
        alive = false;
        break;
      }
      tc_fence_after_sync();
      if (tile + 1 == tile1) DECODE_STAMP(p, 6, warp == 6 && lane == 0);
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(buf * BN);
      const int krow = tile * kTileM + q * 32 + lane;
      // a chunk of the finished sum: the last piece's accumulator, with what the others left
      auto load16 = [&](int c, uint32_t (&r)[16]) {
        tmem_ld_32x16(taddr + static_cast<uint32_t>(c), r);
        if constexpr (kPieces) {
          if (summed) {
            uint32_t w[16];
            tmem_ld_32x16(tsum + static_cast<uint32_t>(c), w);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = add_f32(w[j], r[j]);
            return;
          }
        }
        tmem_ld_wait();
      };
      if (splits == 1 && p.Nk > 16 && !kPieces) {
        for (int c = 0; c < p.Nk; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32(taddr + static_cast<uint32_t>(c), r);
          tmem_ld_wait();
          if (c + 32 >= p.Nk) hand_back();
          if (krow < p.Mk) decode_store_chunk<32>(e, r, krow, c, min(32, p.Nk - c));
        }
      } else if (splits == 1 && kPieces) {
#pragma unroll 1
        for (int c = 0; c < p.Nk; c += 16) {
          uint32_t r[16];
          load16(c, r);
          if (c + 16 >= p.Nk) hand_back();
          if (krow < p.Mk) decode_store_chunk<16>(e, r, krow, c, min(16, p.Nk - c));
        }
      } else if (splits == 1) {
        uint32_t r[16];
        load16(0, r);
        if (tile + 1 == tile1) DECODE_STAMP(p, 8, warp == 6 && lane == 0);
        hand_back();
        if (krow < p.Mk) decode_store_chunk<16>(e, r, krow, 0, p.Nk);
        if (tile + 1 == tile1) DECODE_STAMP(p, 10, warp == 6 && lane == 0);
      } else {
        for (int c = 0; c < nchunks; ++c) {
          uint32_t r[16];
          load16(c * 16, r);
          // this lane's 64 bytes of the unit, 16-byte pieces XOR-swizzled over pairs of lanes
          // (rows are 64 bytes apart: without it every other lane would meet the same banks)
          const int u = q + 4 * c, owner = u % splits, slot = u / splits;
          const uint32_t dst = map_to_cta(
              red_base + static_cast<uint32_t>((slot * splits + rank) * kDecodeUnitBytes + lane * 64),
              static_cast<uint32_t>(owner));
          const uint32_t bar = map_to_cta(red_bar(slot), static_cast<uint32_t>(owner));
          const uint32_t swz = static_cast<uint32_t>(lane >> 1) & 3u;
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j)
            st_async_v4(dst + ((j ^ swz) << 4), r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3], bar);
        }
        hand_back();
      }
      if (++buf == 2) { buf = 0; acc_ph ^= 1u; }
    }
    if (splits > 1) cluster_arrive();  // nothing more leaves this warp for another CTA
    if (splits > 1 && alive) {
      // the units this CTA owns: the pieces added in ascending k order, then the epilogue
      const int units = decode_reduce_units(p.Nk);
      for (int slot = warp - 6; rank + slot * splits < units; slot += 4) {
        const bool got = mbar_wait_bounded(red_bar(slot), 0, abort_flag, budget_ns);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0) {
            leave_error(p.error, kErrEpilogueWait);
            *abort_flag = 1;
          }
          break;
        }
        const int u = rank + slot * splits;
        const uint32_t swz = static_cast<uint32_t>(lane >> 1) & 3u;
        uint32_t src = red_base + static_cast<uint32_t>(slot * splits * kDecodeUnitBytes + lane * 64);
        float acc[16];
        for (int pc = 0; pc < splits; ++pc, src += kDecodeUnitBytes) {
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j) {
            float4 v;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                         : "r"(src + ((j ^ swz) << 4)));
            acc[4 * j] = pc == 0 ? v.x : __fadd_rn(acc[4 * j], v.x);
            acc[4 * j + 1] = pc == 0 ? v.y : __fadd_rn(acc[4 * j + 1], v.y);
            acc[4 * j + 2] = pc == 0 ? v.z : __fadd_rn(acc[4 * j + 2], v.z);
            acc[4 * j + 3] = pc == 0 ? v.w : __fadd_rn(acc[4 * j + 3], v.w);
          }
        }
        uint32_t r[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(acc[j]);
        const int krow = tile0 * kTileM + (u & 3) * 32 + lane, kcol0 = (u >> 2) * 16;
        if (krow < p.Mk) decode_store_chunk<16>(e, r, krow, kcol0, min(16, p.Nk - kcol0));
      }
    }
  }

  DECODE_STAMP(p, 7, warp == 6 && lane == 0);
  if (splits > 1 && *abort_flag != 0 && threadIdx.x == 0) {
    // pieces that were on their way when this CTA gave up waiting for them: time to land
    const uint64_t t_end = global_timer_ns() + 200000;
    while (global_timer_ns() < t_end) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncwarp();
  if (splits > 1) {
    // No CTA leaves while another may still send to it (which the waits above imply, unless one
    // of them gave up).
    if (warp < 6) {
      cluster_wait();
      cluster_arrive();
    }
    cluster_wait();
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, static_cast<uint32_t>(p.tmem_cols));
}

}  // namespace b200
