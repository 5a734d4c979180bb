// Small HBM-bound helper kernels around the tensor-core GEMM:
//   * relayout_scales_kernel  -- row-major E8M0 scales -> tile-ordered atoms
//   * reduce_epilogue_kernel  -- split-k slab reduction in fixed slice order +
//                                epilogue; with zero slabs it is the k == 0 path
//   * repack_rows_kernel      -- copies operands whose base / leading dimension
//                                TMA cannot address into a 16-byte aligned pitch
#pragma once

#include "epilogue.cuh"
#include "gemm_params.h"
#include "ptx_sm100.cuh"

namespace b200 {

// Self-test of the bounded-wait path: one warp waits, with the given budget, on an mbarrier
// that nothing ever arrives on.  The wait gives up when the budget is spent, the warp
// records kErrProducerWait in the device error word exactly as the GEMM kernels' roles do,
// and the kernel returns normally: nothing hangs, traps or faults.
__global__ void wait_timeout_probe_kernel(int32_t* error, uint32_t budget_us) {
  __shared__ __align__(8) uint64_t bar;
  __shared__ int abort_flag;
  const uint32_t bar_addr = smem_u32(&bar);
  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(bar_addr, 1);
    fence_mbar_init();
  }
  __syncwarp();
  const bool done = mbar_wait_bounded(bar_addr, 0, &abort_flag, static_cast<uint64_t>(budget_us) * 1000ull);
  if (!__all_sync(0xffffffffu, done) && threadIdx.x == 0) leave_error(error, kErrProducerWait);
}

// Scale layout consumed by tcgen05.cp (32x128b.warpx4) + block-scaled MMAs.
// The CPU library reads scales[row*ld + kk/32] directly while packing
// (gemm/threadblock/mma_policy_mx.h:213,219,242,248).  Here, for every tile of
// `tile_rows` rows (128 on the MMA-M side, BN on the N side) and every pipeline
// stage of `bps` scale blocks (4 for fp8: 128 elements, 8 for fp4: 256
// elements), the stage chunk is an array of 512-byte atoms
//     atom (ka, nb), ka < bps/4, nb < ceil(tile_rows/128)
//     byte (r%32)*16 + ((r%128)/32)*4 + (kb%4)
// for row r of the tile (nb = r/128) and scale block kb = stage*bps + ka*4 + kb%4.
// One warp writes one atom (512 contiguous bytes); each lane gathers the 4x4
// bytes of rows l, l+32, l+64, l+96.  Out-of-range rows / blocks get 127
// (1.0): the zero-filled operand padding must never meet a NaN scale, and
// caller memory past ceil(k/32) entries of a row is never read.
struct ScaleLayout {
  int rows, kblocks;       // valid rows, ceil(k/32)
  int ld;                  // leading dimension of the source (entries)
  int tile_rows, nb128;    // rows per tile, 128-row atoms per tile
  int bps, ka;             // scale blocks per stage, atoms along k per stage
  int tiles, stages;       // number of row tiles, pipeline stages along k
};

// One warp re-lays-out four consecutive atoms along k of one 128-row group: lane l
// reads 16 scale bytes (four 4-block quads) of rows l, 32 + l, 64 + l and 96 + l and
// writes one 16-byte piece (its row of each of the four 32-row sub-groups) per atom,
// so every atom is written as one coalesced 512-byte line.  Rows, k blocks and tile
// rows outside the matrix read as 0x7F (scale 1.0; the operand data there is zero).
__device__ __forceinline__ void relayout_four_atoms(const uint8_t* __restrict__ src,
                                                    uint8_t* __restrict__ dst, const ScaleLayout& L,
                                                    int64_t w, int lane) {
  const int k_atoms = L.stages * L.ka;
  const int k_groups = (k_atoms + 3) >> 2;
  const int kg = static_cast<int>(w % k_groups);
  const int64_t rg = w / k_groups;  // (tile, nb)
  const int nb = static_cast<int>(rg % L.nb128);
  const int tile = static_cast<int>(rg / L.nb128);
  const int kb0 = kg * 16;
  const bool vec_ok = (L.ld % 16 == 0) && ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) &&
                      kb0 + 15 < L.kblocks;
  uint32_t words[4][4];  // [sub-group][atom]
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const int r_in_tile = nb * 128 + g * 32 + lane;
    const int row = tile * L.tile_rows + r_in_tile;
    const bool row_ok = r_in_tile < L.tile_rows && row < L.rows;
    const uint8_t* s = src + static_cast<int64_t>(row) * L.ld + kb0;
    if (row_ok && vec_ok) {
      const uint4 v = *reinterpret_cast<const uint4*>(s);
      words[g][0] = v.x; words[g][1] = v.y; words[g][2] = v.z; words[g][3] = v.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t word = 0;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int kb = kb0 + 4 * j + t;
          const uint32_t byte = (row_ok && kb < L.kblocks) ? s[4 * j + t] : 127u;
          word |= byte << (8 * t);
        }
        words[g][j] = word;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int kq = kg * 4 + j;
    if (kq < k_atoms) {
      const int stage = kq / L.ka, ka = kq % L.ka;
      const int64_t atom_off =
          ((static_cast<int64_t>(tile) * L.stages + stage) * (L.ka * L.nb128) + ka * L.nb128 + nb) * 512;
      *reinterpret_cast<uint4*>(dst + atom_off + lane * 16) =
          make_uint4(words[0][j], words[1][j], words[2][j], words[3][j]);
    }
  }
}

__host__ __device__ inline int64_t relayout_work_items(const ScaleLayout& L) {
  return static_cast<int64_t>(L.tiles) * L.nb128 * ((L.stages * L.ka + 3) / 4);
}

// One launch re-lays-out up to two scale arrays (the A-side and B-side operands
// of one GEMM).  The GEMM kernel that consumes the result may be launched with
// programmatic stream serialization: its prologue then overlaps this kernel, and
// its TMA producer waits (griddepcontrol.wait) before the first scale load.
__global__ void relayout_scales_kernel(const uint8_t* __restrict__ src0, uint8_t* __restrict__ dst0,
                                       ScaleLayout L0, const uint8_t* __restrict__ src1,
                                       uint8_t* __restrict__ dst1, ScaleLayout L1) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // launched with programmatic stream serialization itself: the GEMM before it may still be
  // reading the atoms this kernel is about to overwrite
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int64_t items0 = relayout_work_items(L0);
  const int64_t items1 = src1 ? relayout_work_items(L1) : 0;
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t w = warp0; w < items0 + items1; w += nwarps) {
    if (w < items0) {
      relayout_four_atoms(src0, dst0, L0, w, lane);
    } else {
      relayout_four_atoms(src1, dst1, L1, w - items0, lane);
    }
  }
}

// D = epilogue(sum_s slab_s) with the slabs added in slice order
// ((w0 + w1) + w2) + ..., as the CPU library's reduce_splitk does
// (gemm/kernel/run_blocked.h:40-75); slices == 0 is its write_zero_k (:30-36).
// A slab is stored column by column (the accumulator's lanes are rows, so the GEMM writes
// 128 contiguous bytes per instruction; by rows of D it wrote 16 bytes to each of 32 lines).
// A block reads 32 rows x kCols columns of every slab - kCols / 8 elements per thread, the words of several
// slabs in flight - and turns them in shared memory where D's rows are contiguous.  Small outputs take
// kCols = 8, many blocks: bound by the latency of those reads and by the gap between two launches, which
// programmatic stream serialization hides: 192 x 320 x 16384 u8 x s8, both kernels, 12.4 us in
// 22 slices (13.5 without), 11.1 in 8.  Large ones take 32: with 8 a row of D is written 32 bytes at a time (GEMM and reduction,
// kCols = 8 / 32: 640 x 1024 x 16384 in 3 slices 20.9 / 18.2 us, 1024 x 2048 x 16384 in 4 53.1 / 42.2,
// 2048 x 2048 x 8192 in 2 76.7 / 55.7; 1000 x 300 x 8192 e4m3 in 8 20.9 / 22.5, too few blocks).
template <bool kInt, int kCols>
__global__ void __launch_bounds__(256) reduce_epilogue_kernel(EpilogueParams e, const uint32_t* ws, int slices, int Mk,
                                                              int Nk) {
  constexpr int kPer = kCols / 8;           // columns per warp
  constexpr int kFlight = kPer == 1 ? 8 : 4;  // slabs whose words are in flight together
  __shared__ uint32_t turn[kCols][33];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int row_tiles = (Mk + 31) / 32, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tiles = static_cast<int64_t>(row_tiles) * ((Nk + kCols - 1) / kCols), slab = static_cast<int64_t>(Mk) * Nk;
  const bool by_rows = e.d_sr != 1;
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the slabs are written
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int row0 = static_cast<int>(t % row_tiles) * 32, col0 = static_cast<int>(t / row_tiles) * kCols;
    uint32_t acc[kPer];
#pragma unroll
    for (int c = 0; c < kPer; ++c) acc[c] = 0;
    if (slices > 0 && row0 + lane < Mk) {
      const uint32_t* w = ws + (static_cast<int64_t>(col0 + warp) * Mk + row0 + lane);
      for (int s0 = 0; s0 < slices; s0 += kFlight) {
        uint32_t v[kFlight][kPer];
#pragma unroll
        for (int j = 0; j < kFlight; ++j)
#pragma unroll
          for (int c = 0; c < kPer; ++c)
            v[j][c] = s0 + j < slices && col0 + warp + 8 * c < Nk ? __ldcg(w + (s0 + j) * slab + static_cast<int64_t>(8 * c) * Mk) : 0u;
#pragma unroll
        for (int j = 0; j < kFlight; ++j) {
          if (s0 + j >= slices) break;
#pragma unroll
          for (int c = 0; c < kPer; ++c) {
            if (s0 + j == 0) {
              acc[c] = v[0][c];
            } else if constexpr (kInt) {
              acc[c] += v[j][c];
            } else {
              acc[c] = __float_as_uint(__fadd_rn(__uint_as_float(acc[c]), __uint_as_float(v[j][c])));
            }
          }
        }
      }
    }
    if (by_rows) {
#pragma unroll
      for (int c = 0; c < kPer; ++c) turn[warp + 8 * c][lane] = acc[c];
      __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < kPer; ++c) {
      int krow = row0 + lane, kcol = col0 + warp + 8 * c;
      if (by_rows) {
        const int i = static_cast<int>(threadIdx.x) + 256 * c;
        krow = row0 + i / kCols;
        kcol = col0 + i % kCols;
        acc[c] = turn[i % kCols][i / kCols];
      }
      if (krow < Mk && kcol < Nk)
        static_cast<uint32_t*>(e.D)[krow * e.d_sr + kcol * e.d_sc] = epilogue_element<kInt>(e, acc[c], krow, kcol);
    }
    if (by_rows) __syncthreads();  // (the next tile overwrites it)
  }
}

// An operand that TMA cannot address, and the 16-byte aligned copy of it that the GEMM reads.
// With `mask_last_high_nibble` the high nibble of each row's last byte is cleared (packed
// fp4 with an odd k: that nibble belongs to element k, which is outside the problem).
struct RepackJob {
  const uint8_t* src;  // any alignment
  uint8_t* dst;        // 16-byte aligned, pitch a multiple of 16; may be src (nibble mask only)
  int64_t src_pitch, dst_pitch;
  int rows, row_bytes, mask_last_high_nibble;
};
__host__ __device__ inline uint32_t repack_row_pieces(const RepackJob& j) {  // 512-byte pieces, one per warp
  return (static_cast<uint32_t>(j.row_bytes) + 511u) / 512u;
}
__host__ __device__ inline int64_t repack_work_items(const RepackJob& j) {
  return static_cast<int64_t>(j.rows) * repack_row_pieces(j);
}

// Lane l of the warp writes bytes [512 piece + 16 l, + 16) of a row.
__device__ __forceinline__ void repack_piece(const RepackJob& j, uint32_t item, int lane) {
  const uint32_t pieces = repack_row_pieces(j);
  const uint32_t row = item / pieces;
  const int c0 = static_cast<int>((item - row * pieces) * 512u) + lane * 16;
  const int left = j.row_bytes - c0;  // bytes of the row from here on
  if (left <= 0) return;
  const uint8_t* s = j.src + static_cast<int64_t>(row) * j.src_pitch + c0;
  const uint8_t* end = j.src + static_cast<int64_t>(j.rows - 1) * j.src_pitch + j.row_bytes;
  const uint32_t off = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(s) & 3u);
  uint32_t w[5] = {0, 0, 0, 0, 0};
  if (s - off >= j.src && s - off + 20 <= end) {
    // five aligned words hold the 16 bytes wherever they start; all lie inside the operand
    const uint32_t* a = reinterpret_cast<const uint32_t*>(s - off);
#pragma unroll
    for (int i = 0; i < 5; ++i) w[i] = a[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w[i] = __funnelshift_r(w[i], w[i + 1], off * 8u);
      const int valid = left - 4 * i;  // bytes of this word that belong to the row
      if (valid < 4) w[i] = valid <= 0 ? 0u : w[i] & ((1u << (8 * valid)) - 1u);
    }
  } else {  // the operand's first and last bytes
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (i < left) w[i >> 2] |= static_cast<uint32_t>(s[i]) << (8 * (i & 3));
  }
  if (j.mask_last_high_nibble && left <= 16) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (i == left - 1) w[i >> 2] &= ~(0xF0u << (8 * (i & 3)));
  }
  *reinterpret_cast<uint4*>(j.dst + static_cast<int64_t>(row) * j.dst_pitch + c0) = make_uint4(w[0], w[1], w[2], w[3]);
}

// Copies up to two operands (j1.rows == 0: one) into 16-byte aligned rows.  Bound by HBM and
// L2: every warp reads 512 contiguous bytes in aligned 4-byte words and writes them in 16-byte
// ones.  One launch for both operands, and programmatic stream serialization on both sides
// of it (the GEMM's prologue runs beside it): 3.5 + 5.3 MB in 6 us.
__global__ void __launch_bounds__(256) repack_rows_kernel(RepackJob j0, RepackJob j1) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the GEMM before may still read the old copies
  const uint32_t items0 = static_cast<uint32_t>(repack_work_items(j0));
  const uint32_t items = items0 + (j1.rows > 0 ? static_cast<uint32_t>(repack_work_items(j1)) : 0u);
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < items; w += warps) {
    if (w < items0) {
      repack_piece(j0, w, static_cast<int>(threadIdx.x & 31u));
    } else {
      repack_piece(j1, w - items0, static_cast<int>(threadIdx.x & 31u));
    }
  }
}

}  // namespace b200
