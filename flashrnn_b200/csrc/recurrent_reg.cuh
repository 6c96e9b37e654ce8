// Shape rules and device helpers of the register-resident recurrence kernels (recurrent_reg_fwd.cuh, recurrent_reg_bwd.cuh).
//
// A step of a narrow head is a product of a [GR*U x D] slice of R with a [D x 8] operand: 8 batch rows, one warp-level
// m16n8k16 column tile. tcgen05.mma spends about 79 cycles per 128x16x16 instruction whatever the 8 columns need, and its
// result comes back through tensor memory and shared memory (commit, tcgen05.ld, gate buffer, barrier). Here the slice of
// R lives in the registers of the warps as mma.sync fragments for the whole sequence, the accumulators of a unit's gates
// land in the registers of the thread that runs the cell, and nothing but the operand itself passes through shared memory.
//
// A warp has 4 units (a 16-row tile holds their four gates), so that a thread has one item (unit, batch row) per column tile and an SM
// sub-partition two warps: a lone warp issues an instruction every 4.5 cycles, and of 8 units per warp the cell, the staging and the
// publication were twice as many instructions on the chain of a step (LSTM B8 N3 D256, us per step forward / backward: 0.80 / 0.89
// against 0.64 / 0.66).
#pragma once

#include "frnn_common.cuh"

namespace frnn {

constexpr int kRegRows = 8;           // batch rows of one column tile of an mma; a group has one, two or (clusters of 5 CTAs and more) three
constexpr int kRegMaxRows = 24;
constexpr int kRegNoRoom = -100;      // not taken: too many waves, or outputs off the 16-byte grid
constexpr int kRegTaken = -101;       // answer to a question: the call would run here

// Widths of these kernels: all multiples of 16 up to 256, multiples of 32 up to 512. One CTA holds a head of 16, 32 or 48 units
// whole; other widths run as a cluster of CTAs with 32 units, the last of which has 16 units where D is an odd multiple of 16.
// At 64 units one CTA's warps would share the schedulers and its I/O warp move two 32-unit tiles per step: with 8 units per warp, LSTM, 8
// rows, fp32 Wx, 0.85 + 1.19 us per step forward + backward against 0.63 + 0.68 as a cluster of two. CTAs of 16 units (clusters of
// 16 at 256) were no faster either: forward 0.68 against 0.67.
inline bool reg_width(int D) { return D % 16 == 0 && (D <= 256 || (D % 32 == 0 && D <= 512)); }
inline bool reg_local(int D) { return D < 64; }

inline int reg_batch_tiles(int B, int rows) { return (B + rows - 1) / rows; }
// Compile-time bound on the 16-wide k tiles of the width: exact for one CTA, even in a cluster (operands are fetched 32 k at a
// time), multiples of 4 from 288 units on (fewer instantiations; the tiles past the head are zero).
inline int reg_k_tiles(int D) { return reg_local(D) ? D / 16 : (D <= 256 ? (D + 31) / 32 * 2 : (D + 63) / 64 * 4); }

// Staged tiles (Wx, cache, states, gradients): per chunk of 32 units of the CTA (wide heads: the units it owns) and per plane (gate or
// state) the batch rows of the group, rows of 32, 64 or 128 bytes under the TMA swizzle of that span. The threads of a warp
// read 4 units of 8 rows at once: un-swizzled these rows would share their banks.
constexpr int kRegChunk = 32;
// The swizzle follows address bits: planes start at multiples of 8 rows.
__host__ __device__ constexpr int reg_round_1k(int bytes) { return (bytes + 1023) & ~1023; }
// Dynamic shared memory that every launcher asks for, whatever its call needs: the attribute belongs to the kernel, and a
// thread that set it to the need of its own call (26 KB for bf16 inference at 256 units) could take it from one that is
// about to launch (49 KB for fp32 training).
constexpr int kRegSmemLimit = 220 * 1024;
// Tiles travel several steps at a time: a transfer is 4 steps of every plane, or fewer where 4 would not let as many CTAs share an SM
// as the registers do, and two of them are in flight in either direction. A warp waits for its input and reports its output once
// per transfer: waiting, fences, arrivals and the bookkeeping around them are instructions on the chain of a step.
constexpr int kRegSlots = 2;
inline int reg_transfer_steps(int fixed_bytes, int step_bytes, int blocks) {
  const int limit = blocks == 1 ? kRegSmemLimit - 2 * kRegSlots * 1024 : 224 * 1024 / blocks;  // less what rounding adds
  int steps = 4;
  while (steps > 1 && fixed_bytes + kRegSlots * steps * step_bytes > limit) --steps;
  return steps;
}

// Modes of the step loops. Forward: any outputs and the hooks, any outputs, those of a training call, the same with h clipped, a whole fp32
// history alone, fp32 hidden states alone, bf16 snapshots alone, nothing but the carry. Backward: options and hooks, options, neither.
// The loops of training calls and whole histories have kernels without the others (EXTRA), where each of them has the hooks' loop beside it:
// registers are assigned to a kernel as a whole, and fragments that were spilled for the sake of another loop were up to 8 % (LSTM
// B64 T48 N1 D320 backward 49.1 us against 46.4, Elman B280 D448 inference 120 / 111).
enum : int { kRegHooks = 0, kRegAny, kRegTrain, kRegClipped, kRegPlain, kRegHidden, kRegNarrow, kRegLast };

// Wide heads (recurrent_wide_*.cuh): slots of the exchange in global memory, steps between two fences.
constexpr int kWideSlots = 64, kWideFence = 8;
inline int wide_slots(int T) { return T < kWideSlots ? T : kWideSlots; }

// Tensor map with the dimensions (unit of the head, head, batch row, plane, step). A box that reaches past the head, the
// batch or the steps is filled with zeros on the way in and cut off on the way out.
inline int reg_tile_map(CUtensorMap* map, const void* base, int es, int D, int N, int B, int planes, int steps,
                        uint64_t batch_stride, uint64_t plane_stride, uint64_t step_stride, int box_planes, int chunk, int rows, int box_steps) {
  const uint64_t dims[5] = {static_cast<uint64_t>(D), static_cast<uint64_t>(N), static_cast<uint64_t>(B),
                            static_cast<uint64_t>(planes), static_cast<uint64_t>(steps)};
  const uint64_t strides[4] = {static_cast<uint64_t>(D) * es, batch_stride * es, plane_stride * es, step_stride * es};
  const uint32_t box[5] = {static_cast<uint32_t>(chunk), 1u, static_cast<uint32_t>(rows), static_cast<uint32_t>(box_planes), static_cast<uint32_t>(box_steps)};
  return make_tensor_map_strided(map, base, es, 5, dims, strides, box, chunk * es);
}

// Clusters of `width` CTAs (or plain CTAs: 1) that run at once, or minus a cudaError_t. Raises the kernel's shared-memory limit and allows
// it clusters of 16; what it asks the driver for is remembered.
int reg_capacity(const void* kern, const cudaLaunchConfig_t& cfg, int width);
// 0 if a launch of `groups` clusters is taken, kRegNoRoom if not, else a cudaError_t. `rival_groups` > 0: plain CTAs may also run in several
// waves, as long as these are not more than 4/3 of the waves of so many 16-row groups of the tcgen05 kernels.
int reg_room(const void* kern, const cudaLaunchConfig_t& cfg, int width, long long groups, long long rival_groups, int D);

// How the tcgen05 kernels would run a call of at most 512 units: batch rows of a group, waves (0: unknown). Where these need a second
// wave, register groups of more than 8 rows are always faster.
struct RegRival { int rows, waves; };
RegRival reg_rival(bool backward, int cell, int wx_bf16, int N, int B, int D);

// Whether a call runs the kernels with the other loops.
template <int CELL>
bool reg_extra(const FwdParams& p, int hist_states, bool has_cache) {
  const bool train = p.hbf != nullptr && (has_cache || CELL == kElman), plain = p.hbf == nullptr && !has_cache;
  return hist_states != CellTraits<CELL>::S || p.out_bf16 != 0 || p.fwd_clip < INFINITY || !(train || plain);
}
inline bool reg_extra(const BwdParams& p) { return p.cut_recurrent != 0 || p.grad_clip > 0.0f || p.slstm_v1 != 0; }

#ifdef __CUDACC__
__device__ __forceinline__ void reg_report(int* err, int code, int detail) {
  if (atomicCAS(err, 0, code) == 0) {
    err[1] = detail;
    err[2] = static_cast<int>(blockIdx.x);
  }
  __threadfence();
}

// Byte offset of (batch row, unit of the chunk) in a plane of the staged tiles: rows of CHUNK * ES bytes, 16-byte blocks
// permuted as the TMA swizzle of that span does (none at 16 bytes).
template <int ES, int CHUNK>
__device__ __forceinline__ uint32_t reg_tile_offset(int row, int unit) {
  constexpr int span = CHUNK * ES;
  const int x = span == 128 ? row & 7 : (span == 64 ? (row >> 1) & 3 : (span == 32 ? (row >> 2) & 1 : 0));
  return static_cast<uint32_t>(row * span) + (static_cast<uint32_t>(unit * ES) ^ static_cast<uint32_t>(x << 4));
}
__device__ __forceinline__ float lds_f32(uint32_t a) { float v; asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) { uint16_t v; asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a)); return v; }
__device__ __forceinline__ void sts_f32(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void sts_u16(uint32_t a, uint32_t v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"(static_cast<uint16_t>(v)) : "memory"); }
__device__ __forceinline__ uint32_t bf16_bits(float v) { return static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v))); }

// The first of two operand buffers [column tile][k][8 batch rows] from the initial states (row 0 of the head, `row` floats from batch row
// to batch row), the second one zero. A word is two batch rows of one k; neighbouring threads take neighbouring k.
template <int NB, int KT>
__device__ __forceinline__ void reg_fill_operand(uint8_t* buf, const float* initial, size_t row, int b0, int B, int K, int tid, int threads) {
  constexpr int kWords = NB * KT * 64;
#pragma unroll 4
  for (int i = tid; i < kWords; i += threads) {
    const int k = i % (KT * 16), pair = i / (KT * 16), b = b0 + 2 * pair;  // pair: column tile * 4 + rows of it / 2
    const float* const src = initial + static_cast<size_t>(b) * row + k;
    const float lo = k < K && b < B ? __ldg(src) : 0.0f, hi = k < K && b + 1 < B ? __ldg(src + row) : 0.0f;
    reinterpret_cast<uint32_t*>(buf)[(pair >> 2) * (KT * 64) + k * 4 + (pair & 3)] = pack_bf16x2(lo, hi);
  }
  for (int i = tid; i < kWords / 4; i += threads) reinterpret_cast<uint4*>(buf + kWords * 4)[i] = make_uint4(0u, 0u, 0u, 0u);
}

// A fragments of a 16-row tile, K k of which count. Row r of the tile is `base` + (r / UPW) * gate + (r % UPW) * stride (elements) while
// its gate r / UPW < GR, else zeros. Rows on the 16-byte grid come 64 k at a time through 2 KB of the warp's own shared memory:
// 4 loads, 4 stores and an ldmatrix per k tile, where word by word a thread has four loads per k tile, all of them
// unrolled. Prologue in cycles, word by word / this: LSTM D256 N3 13.0 k / 10.5 k, D128 N4 9.0 k / 5.8 k, D768 8.9 k / 6.5 k; LSTM B4 T16
// N1 D768 38.2 us / 37.4.
constexpr int kRegScratch = 2048;
template <int KT, int UPW, int GR>
__device__ __forceinline__ void reg_load_rows(const __nv_bfloat16* base, size_t gate, size_t stride, int K, uint32_t scratch, int lane,
                                              bool aligned, uint32_t (&a)[KT][4]) {
  if (aligned) {
    constexpr int CHUNKS = (KT + 3) / 4;
    const int r0 = lane >> 3, col = lane & 7;  // this lane's piece: rows r0 + 4 j, 8 k
    uint4 v[CHUNKS][4];
#pragma unroll
    for (int m = 0; m < CHUNKS; ++m)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int g = 4 * j / UPW, u = UPW == 4 ? r0 : r0 + 4 * (j & 1);
        v[m][j] = g < GR && m * 64 + col * 8 < K ? __ldg(reinterpret_cast<const uint4*>(base + g * gate + u * stride + m * 64 + col * 8))
                                                 : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
    for (int m = 0; m < CHUNKS; ++m) {
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = r0 + 4 * j;
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(scratch + r * 128 + ((col ^ (r & 7)) << 4)), "r"(v[m][j].x), "r"(v[m][j].y),
                     "r"(v[m][j].z), "r"(v[m][j].w) : "memory");
      }
      __syncwarp();
      const int r = ((lane >> 3) & 1) * 8 + (lane & 7);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (4 * m + i < KT) ldsm_x4(scratch + r * 128 + (((2 * i + (lane >> 4)) ^ (r & 7)) << 4), a[4 * m + i]);
    }
    // TMA writes these bytes next: ordinary accesses and those of the async proxy are ordered by a proxy fence, which the caller's
    // cluster barrier alone is not.
    fence_proxy_async_smem();
  } else {
    const int q = lane >> 2, c = lane & 3;
#pragma unroll
    for (int kt = 0; kt < KT; ++kt)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int row = q + 8 * (r & 1), g = row / UPW, k = kt * 16 + 8 * (r >> 1) + 2 * c;
        a[kt][r] = g < GR && k < K ? __ldg(reinterpret_cast<const uint32_t*>(base + g * gate + row % UPW * stride + k)) : 0u;
      }
  }
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
