// Shape rules and device helpers of the register-resident recurrence kernels (recurrent_reg_fwd.cu, recurrent_reg_bwd.cu).
//
// A step of a narrow head is a product of a [GR*U x D] slice of R with a [D x 8] operand: 8 batch rows, one warp-level
// m16n8k16 column tile. tcgen05.mma spends about 79 cycles per 128x16x16 instruction whatever the 8 columns need, and its
// result comes back through tensor memory and shared memory (commit, tcgen05.ld, gate buffer, barrier). Here the slice of
// R lives in the registers of the warps as mma.sync fragments for the whole sequence, the accumulators of a unit's gates
// land in the registers of the thread that runs the cell, and nothing but the operand itself passes through shared memory.
#pragma once

#include "frnn_common.cuh"

namespace frnn {

constexpr int kRegUnitsPerWarp = 8;
constexpr int kRegRows = 8;           // batch rows of a group: the column extent of one mma
constexpr int kRegClusterUnits = 32;  // units of a CTA where a group is a thread-block cluster
constexpr int kRegNoRoom = -100;      // not taken: too many waves, or outputs off the 16-byte grid

// Widths of these kernels: all multiples of 16 up to 256. One CTA holds a head of 16, 32 or 48 units whole; other widths run as
// a cluster of ceil(D / 32) CTAs, the last of which has 16 units where D is an odd multiple of 16.
// At 64 units one CTA's 8 warps share each scheduler two by two and its I/O warp moves two 32-unit tiles per step: LSTM, 8
// rows, fp32 Wx, 0.85 + 1.19 us per step forward + backward against 0.63 + 0.68 as a cluster of two; Elman, 16 rows x 12
// heads, 0.76 + 0.81 us.
inline bool reg_width(int D) { return D % 16 == 0 && D <= 256; }
inline bool reg_local(int D) { return D < 64; }

inline int reg_batch_tiles(int B) { return (B + kRegRows - 1) / kRegRows; }
// Compile-time bound on the 16-wide k tiles of the width (even: operands are fetched 32 k at a time).
inline int reg_k_tiles(int D) { return (D + 31) / 32 * 2; }

// Staged tiles (Wx, cache, states, gradients): per 32 units of the CTA and per plane (gate or state) 8 batch rows of 32
// units, rows of 64 bytes (16-bit) or 128 bytes (32-bit) under the TMA swizzle of that span. The threads of a warp read 8
// units of the batch rows 0, 2, 4, 6 (or 1, 3, 5, 7) at once: un-swizzled these rows share their banks, four ways.
constexpr int kRegChunk = 32;
// The swizzle follows address bits: planes of 32-bit values start at multiples of 1 KB, of 16-bit values at 512 bytes.
__host__ __device__ inline int reg_round_1k(int bytes) { return (bytes + 1023) & ~1023; }
inline int reg_chunks(int U) { return (U + kRegChunk - 1) / kRegChunk; }
constexpr int kRegMaxStages = 4;
// Dynamic shared memory that every launcher asks for, whatever its call needs: the attribute belongs to the kernel, and a
// thread that set it to the need of its own call (26 KB for bf16 inference at 256 units) could take it from one that is
// about to launch (49 KB for fp32 training).
constexpr int kRegSmemLimit = 220 * 1024;
// Steps in flight for a launch that needs so much shared memory with four and with three stages: four, or three where only that
// lets two CTAs share an SM (heads of 48 units with fp32 Wx). With two, a step's tile was fetched only when the step before had
// been staged, and the sLSTM backward, whose registers allow one CTA per SM anyway, gained nothing: forward and backward, B64
// T128 N16 D48 fp32, sLSTM 716 us against 611 now (tcgen05 632), LSTM 589 against 559 (565).
inline int reg_stages(int bytes4, int bytes3) { return bytes4 > 110 * 1024 && bytes3 <= 110 * 1024 ? 3 : kRegMaxStages; }
// Slots of staged outputs: a warp that stages step t has read the input tile of step t, which the I/O warp fetched after
// the copies of step t - stages - 1 had read their slot.
constexpr int kRegMaxSlots = kRegMaxStages + 1;

// Tensor map with the dimensions (unit of the head, head, batch row, plane, step). A box that reaches past the head or the
// batch is filled with zeros on the way in and cut off on the way out.
inline int reg_tile_map(CUtensorMap* map, const void* base, int es, int D, int N, int B, int planes, int steps,
                        uint64_t batch_stride, uint64_t plane_stride, uint64_t step_stride, int box_planes) {
  const uint64_t dims[5] = {static_cast<uint64_t>(D), static_cast<uint64_t>(N), static_cast<uint64_t>(B),
                            static_cast<uint64_t>(planes), static_cast<uint64_t>(steps)};
  const uint64_t strides[4] = {static_cast<uint64_t>(D) * es, batch_stride * es, plane_stride * es, step_stride * es};
  const uint32_t box[5] = {static_cast<uint32_t>(kRegChunk), 1u, static_cast<uint32_t>(kRegRows), static_cast<uint32_t>(box_planes), 1u};
  return make_tensor_map_strided(map, base, es, 5, dims, strides, box, kRegChunk * es);
}

// CTAs per SM the register budget is cut for. Two CTAs of 5 warps leave 168 registers a thread: enough up to 128 units of
// contraction (and for the one-gate cell), while wider slices would spill their fragments, 468 bytes at 256. One-CTA backward
// kernels hold the fragments of all gates of a tile (one sum per tile): four-gate cells would spill at four CTAs per SM, sLSTM
// B16 T1024 N24 D32 2133 us forward and backward against 1849 at three.
constexpr int reg_min_blocks(int cell, int kt, bool local, bool backward) {
  return local ? (kt <= 2 ? (backward && (cell == kLSTM || cell == kSLSTM) ? 3 : 4) : (cell == kSLSTM ? 1 : 2)) : (kt <= 8 || cell == kElman ? 2 : 1);
}

// Threads of a CTA: a warp per 8 units (4 in a cluster; up to 32 units with two k tiles, 48 with four) and the I/O warp.
constexpr int reg_max_threads(int kt, bool local) { return local && kt > 2 ? 7 * 32 : 5 * 32; }

constexpr int kRegTaken = -101;       // answer to a question: the call would run here

// 0 if a launch of N heads and B batch rows is taken, in clusters of `width` CTAs or (1) as plain CTAs, kRegNoRoom if not, else
// a cudaError_t. Raises the kernel's shared-memory limit; the capacity it asks the driver for is remembered.
//   Clusters: all groups run at once. A second wave would double the time, where the tcgen05 kernels can take 16 batch rows
//     per group (LSTM B256 N4 D128: 1.66 us per step in two waves against 1.27 forward, 2.13 against 1.64 backward).
//   Plain CTAs (16, 32, 48 units): several share an SM and need no tensor memory, so they pay in waves too; a wave takes about three
//     quarters of one of 16-row tcgen05 groups, of which an SM holds two. Forward and backward, T128, us, against those: LSTM B256
//     N24 D32 569 / 793, GRU 533 / 709, sLSTM 761 / 1063; LSTM B256 N48 D16 625 / 910, B256 N16 D48 1636 / 1928. The other side
//     is the sLSTM with 16 units and fp32 Wx (11 KB a stage, two CTAs per SM): backward B96 N48, two waves against one, 453 / 269,
//     B400, nine against five, 1645 / 1202.
int reg_room(const void* kern, const cudaLaunchConfig_t& cfg, int width, int N, int B, int D);

#ifdef __CUDACC__
template <int ES> constexpr int kRegPlane = kRegRows * kRegChunk * ES;  // bytes of a staged plane

__device__ __forceinline__ void reg_report(int* err, int code, int detail) {
  if (atomicCAS(err, 0, code) == 0) {
    err[1] = detail;
    err[2] = static_cast<int>(blockIdx.x);
  }
  __threadfence();
}

// Byte offset of (batch row, unit of the chunk) in a plane of the staged tiles.
template <int ES>
__device__ __forceinline__ uint32_t reg_tile_offset(int row, int unit) {
  return static_cast<uint32_t>(row * (kRegChunk * ES)) +
         (static_cast<uint32_t>(unit * ES) ^ static_cast<uint32_t>(ES == 4 ? row << 4 : (row >> 1) << 4));
}

// One value of a unit (q of the warp's 8) for the batch rows 2c and 2c + 1, written to its staged plane: 32-bit values as
// they are, 16-bit pairs transposed inside the warp so that a lane stores two units of one row as a word.
__device__ __forceinline__ void reg_stage_f32(uint8_t* plane, int c, int unit, float v0, float v1) {
  *reinterpret_cast<float*>(plane + reg_tile_offset<4>(2 * c, unit)) = v0;
  *reinterpret_cast<float*>(plane + reg_tile_offset<4>(2 * c + 1, unit)) = v1;
}
__device__ __forceinline__ void reg_stage_16(uint8_t* plane, uint32_t offset_q, uint32_t pair) {
  *reinterpret_cast<uint32_t*>(plane + offset_q) = movmatrix_trans(pair);
}

// Four neighbouring lanes hold one 16-byte packet, a word each: afterwards every lane holds all of it.
__device__ __forceinline__ void gather_quad(uint32_t a, int lane, uint32_t (&pk)[4]) {
  const uint32_t b1 = __shfl_xor_sync(0xffffffffu, a, 1);
  const uint32_t lo = (lane & 1) ? b1 : a, hi = (lane & 1) ? a : b1;
  const uint32_t lo2 = __shfl_xor_sync(0xffffffffu, lo, 2), hi2 = __shfl_xor_sync(0xffffffffu, hi, 2);
  pk[0] = (lane & 2) ? lo2 : lo; pk[1] = (lane & 2) ? hi2 : hi;
  pk[2] = (lane & 2) ? lo : lo2; pk[3] = (lane & 2) ? hi : hi2;
}
#endif

}  // namespace frnn
