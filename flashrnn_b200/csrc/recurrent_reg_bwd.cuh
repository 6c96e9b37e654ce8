// Reverse-time recurrence of narrow heads with R in the register file (see recurrent_reg.cuh).
//
// Groups, CTAs and the items of a thread are those of recurrent_reg_fwd.cuh (4 units a warp for every cell). Per step t a thread
//   1. adds up the partial dh_t of its items (fixed order), the external gradient and the pointwise
//      carry, runs the cell backward and writes round_bf16(dg_t) to shared memory for ldmatrix (one CTA barrier),
//   2. multiplies with its warp's fragments of R_slice^T [D x GR*U] (rows = units p of h_{t-1}, k = gate rows of this CTA),
//   3. hands the accumulators to the owners of those units as they lie: two batch rows of a unit, 8 bytes.
// The sums of step 2 run over the same gate rows in the same order as in the tcgen05 kernels, whose CTAs own 32 units (16
// where the width is not a multiple of 32), and step 1 adds them in the same order: every gradient is the same bits, whichever
// kernels a call takes.
//   LOCAL: D / 16 row tiles for D / 4 warps. 16 and 32 units: one sum per tile, which the first warps run; 48 units: three
//          "sources" of 16 units each, a warp for each of the nine (tile, sum) pairs.
//   else:  the sources are the CTAs of the cluster, packets travel by st.async. HALVES (odd multiples of 16): two sums per
//          tile, one for each 16 units of the CTA; the last CTA has units, and a sum, in its first half only.
// The state of step t - 1 stays in registers as the new state of the next iteration, and only the planes that the cell's
// derivative reads are fetched: an LSTM reads one history plane per step where reading both states at t and t - 1 takes four.
//
// Safe reuse: dg is double-buffered because a warp may still read dg_t when another has begun step t - 1; the partial
// sums of a parity are overwritten only after the CTA barrier of the step that read them; a TMA stage is refilled by the I/O
// warp after every warp has staged its outputs of the step that used it.
//
// Bound: the serial chain of a step, as in recurrent_reg_fwd.cuh. LSTM B8 N3 D256, cycles: tiles read, partial sums
// awaited (316) and added 526, cell 83, staging 64, mma and scatter 442; the prologue is 9.5 k.
// us per step before (8 units a warp, a transfer per step) and now: LSTM B8 N3 D256 0.89 / 0.66; LSTM B16 N4 D128 0.78 / 0.58; sLSTM
// there 1.03 / 0.90 (its derivative is the longest); LSTM B8 N1 D64 fp32 0.70 / 0.62; GRU B16 N24 D32 0.71 / 0.46; Elman B16 N12 D64 0.49 /
// 0.35. Against the tcgen05 kernels, which had these before: LSTM B256 N4 D128 (16 rows) 1.68 / 1.38; B8 N1 D384 1.61 / 0.85, D512 1.84 /
// 1.45; B64 N3 D256 (24 rows) 1.77 / 1.06.
#pragma once

#include <type_traits>

#include "recurrent_reg.cuh"

namespace frnn {

namespace {

// History planes the cell's derivative reads: [first, first + count).
template <int CELL> struct HistPlanes;
template <> struct HistPlanes<kLSTM> { static constexpr int first = 1, count = 1; };
template <> struct HistPlanes<kSLSTM> { static constexpr int first = 1, count = 3; };
template <> struct HistPlanes<kGRU> { static constexpr int first = 0, count = 1; };
template <> struct HistPlanes<kElman> { static constexpr int first = 0, count = 1; };

// DENSE: a third CTA on the SM where that saves a wave (see launch_bwd_reg).
template <int CELL, int KT, bool LOCAL, bool HALVES, int NB, bool DENSE = false>
struct BwdRegCfg {
  using CT = CellTraits<CELL>;
  static constexpr int UPW = 4;                         // units of a warp
  static constexpr int U = LOCAL ? KT * 16 : 32, NWARPS = U / UPW, THREADS = (NWARPS + 1) * 32, ROWS = NB * kRegRows;
  static constexpr int MTW = LOCAL ? 1 : (KT + NWARPS - 1) / NWARPS;  // row tiles of a warp
  // Sums of a tile: one over all gate rows of the CTA; in a 48-unit CTA one for units 0 .. 15, 16 .. 31 and 32 .. 47 each, a
  // warp for each of the nine (tile, sum) pairs; with HALVES one for each half of the CTA's units.
  static constexpr int CH = HALVES ? 2 : 1;
  static constexpr int KTW = HALVES || (LOCAL && KT != 2) ? CT::GR : 2 * CT::GR;  // k tiles of a sum
  static constexpr int MAX_SOURCES = LOCAL ? (KT == 3 ? 3 : 1) : (HALVES ? KT : KT / 2);
  static constexpr int DG_BYTES = (CT::GR * U * 16 + 511) / 512 * 512;  // a column tile of dg: [gate row][8 batch rows]
  static constexpr int GCL = CELL == kElman ? 0 : CT::GC;
  static constexpr int HP = HistPlanes<CELL>::first, HS = HistPlanes<CELL>::count;
  static constexpr int PLANE2 = ROWS * kRegChunk * 2, PLANE4 = ROWS * kRegChunk * 4, PLANEC = ROWS * kRegChunk * CT::CES;
  static constexpr int CHUNK = GCL * PLANEC + (HS + CT::S) * PLANE4;  // cache, state of step t - 1, external gradient
  // dg is double-buffered; what follows it starts at a multiple of 1 KB
  static constexpr int DG_ALL = reg_round_1k(2 * NB * DG_BYTES);
  // CTAs per SM the register budget is cut for
  static constexpr int MIN_BLOCKS = LOCAL ? (KT <= 2 ? (NB > 1 || ((CELL == kLSTM || CELL == kSLSTM) && !DENSE) ? 2 : 3) : (CELL == kSLSTM ? 1 : 2))
                                          : (KT <= 8 || CELL == kElman ? 2 : 1);
};

template <int CELL, int KT, bool LOCAL, bool HALVES, int NB, bool DENSE, bool EXTRA>
__global__ void __launch_bounds__(BwdRegCfg<CELL, KT, LOCAL, HALVES, NB, DENSE>::THREADS, BwdRegCfg<CELL, KT, LOCAL, HALVES, NB, DENSE>::MIN_BLOCKS)
frnn_bwd_reg_kernel(const BwdParams p, const float* history, const float* initial, const __grid_constant__ CUtensorMap cache_map,
                    const __grid_constant__ CUtensorMap hist_map,
                    const __grid_constant__ CUtensorMap dhist_map, const __grid_constant__ CUtensorMap dgr_map,
                    const __grid_constant__ CUtensorMap dwx_map, const int wx_bf16, const int own_dwx, const int ring_steps) {
  using Cfg = BwdRegCfg<CELL, KT, LOCAL, HALVES, NB, DENSE>;
  using CT = CellTraits<CELL>;
  constexpr int S = CT::S, MTW = Cfg::MTW, KTW = Cfg::KTW, CH = Cfg::CH, GCL = Cfg::GCL, HP = Cfg::HP, HS = Cfg::HS, U = Cfg::U,
                nwarps = Cfg::NWARPS, UPW = Cfg::UPW, kPlane2 = Cfg::PLANE2, kPlane4 = Cfg::PLANE4;

  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t s_part_bar[2];
  __shared__ __align__(8) uint64_t s_full[kRegSlots];
  __shared__ int s_gave_up;  // a compute warp of this CTA has stopped waiting (the flag in global memory is an L2 round trip away)
  __shared__ __align__(8) uint64_t s_out_full[kRegSlots];  // outputs of a transfer staged by every warp

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane >> 2, c = lane & 3, hi = lane >> 4;
  const long long t_entry = clock64();
  const int D = p.D, N = p.N, T = p.T, B = p.B;
  const int C = LOCAL ? 1 : p.C;
  const int rank = LOCAL ? 0 : static_cast<int>(blockIdx.x % C), gid = blockIdx.x / C;
  const int n = gid % N, b0 = gid / N * Cfg::ROWS;
  const int sources = LOCAL ? Cfg::MAX_SOURCES : (HALVES ? D / 16 : C);
  constexpr int kUnit = kRegRows * 4, kPartTile = U * kUnit, kPartSource = NB * kPartTile;
  const int part_bytes = sources * kPartSource;  // one parity: [source][column tile][unit][8 batch rows] fp32
  constexpr int chunks = (U + kRegChunk - 1) / kRegChunk;
  // A transfer of inputs: per chunk of 32 units the cache, the states of step t - 1 and the external gradient, each for all its steps.
  const int stage_bytes = chunks * ring_steps * Cfg::CHUNK;
  uint8_t* const dgbuf = smem;
  uint8_t* const part = smem + Cfg::DG_ALL;
  uint8_t* const stages = part + 2 * part_bytes;
  uint8_t* const outs = stages + kRegSlots * stage_bytes;
  // Outputs, staged per 32 units: dWx of the steps where it is a tensor of its own, and dg as the dR contraction wants it.
  const int dwx_bytes = own_dwx ? CT::GW * (wx_bf16 ? kPlane2 : kPlane4) : 0;
  const int out_chunk = reg_round_1k(ring_steps * (dwx_bytes + CT::GR * kPlane2)), out_slot = chunks * out_chunk;
  const volatile int* abort_flag = p.err;
  const uint64_t limit = p.wait_limit_ns;
  // hooks of the caller: phase timers; nobody publishes from an iteration on; delays (fp32 Wx: see jitter_stall)
  const bool prof = p.err[3] != 0 && blockIdx.x == 0 && tid == 0;
  const int mute_from = p.err[4] != 0 ? p.err[5] : 0x7fffffff;
  const uint32_t jitter = wx_bf16 ? 0u : static_cast<uint32_t>(p.err[6]);
  const bool hooks = p.err[3] != 0 || p.err[4] != 0 || (jitter != 0u && p.err[7] == 0);  // err[7]: only the I/O warp is late

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&s_part_bar[i]), 1);
    for (int i = 0; i < kRegSlots; ++i) {
      mbar_init(smem_u32(&s_full[i]), 1);
      mbar_init(smem_u32(&s_out_full[i]), nwarps);
    }
    s_gave_up = 0;
    fence_mbar_init();
  }
  for (int i = tid; i < Cfg::DG_ALL / 16; i += blockDim.x)
    reinterpret_cast<uint4*>(dgbuf)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  // the packets carry all 8 columns of a tile whatever the number of batch rows in use
  const uint32_t part_tx = static_cast<uint32_t>(HALVES ? sources * NB * min(U, D - rank * U) * kUnit : part_bytes);
  if (tid == 0 && !LOCAL) {
    mbar_arrive_expect_tx(smem_u32(&s_part_bar[1]), part_tx);              // iteration 1 (the last one if T == 1)
    if (T >= 2) mbar_arrive_expect_tx(smem_u32(&s_part_bar[0]), part_tx);  // iteration 2
  }

  if (warp == nwarps) {
    // ---------------- I/O warp: tiles in, staged outputs out ----------------
    if (!LOCAL) cluster_sync_all();
    if (lane == 0) {
      // A transfer covers the steps t0 .. t0 + ring_steps - 1, t0 a multiple of ring_steps: the first one may reach past the end, none
      // begins before step 0 but the states of step t - 1, whose step -1 is filled with zeros (the compute warps read the initial
      // state instead).
      auto fill = [&](int t0, int s) {
        const uint32_t bar = smem_u32(&s_full[s]);
        mbar_arrive_expect_tx(bar, static_cast<uint32_t>(stage_bytes));
#pragma unroll
        for (int i = 0; i < chunks; ++i) {
          uint32_t dst = smem_u32(stages + s * stage_bytes + i * ring_steps * Cfg::CHUNK);
          const int x = rank * U + i * kRegChunk;
          if (GCL > 0) tma_load_5d(dst, &cache_map, bar, x, n, b0, 0, t0);
          dst += ring_steps * GCL * Cfg::PLANEC;
          tma_load_5d(dst, &hist_map, bar, x, n, b0, HP, t0 - 1);
          dst += ring_steps * HS * kPlane4;
          tma_load_5d(dst, &dhist_map, bar, x, n, b0, 0, t0);
        }
      };
      const int last = (T - 1) / ring_steps * ring_steps;
      for (int i = 0; i < kRegSlots && last - i * ring_steps >= 0; ++i) fill(last - i * ring_steps, i);
      int slot = 0;
      uint32_t phase = 0;
      // Outputs of a transfer staged: released by the CTA's own warps, whose waits have the plain limit, so theirs run out first. The
      // test hook makes this warp late on top of a wait that takes long anyway (the compute warps' stalls see to such waits): on
      // the direct path it costs every step of a run without it up to 80 cycles (Elman B16 N12 D64 backward 0.49 us a step -> 0.57).
      auto staged = [&](int step) -> bool {
        const uint32_t bar = smem_u32(&s_out_full[slot]);
        for (int fast = 0; fast < 64; ++fast)
          if (mbar_try_wait_spin(bar, phase)) return true;
        if (jitter != 0u) jitter_stall(jitter, 32u, static_cast<uint32_t>(step));
        return mbar_wait_bounded<false, true>(bar, phase, 2 * limit, abort_flag);
      };
      for (int t0 = last; t0 >= 0; t0 -= ring_steps) {
        if (!staged(T - 1 - t0)) {
          reg_report(p.err, kErrWaitEmpty, T - 1 - t0);
          break;
        }
        // A warp that gave up on a wait sets the flag before it stages. Then the phase that the barrier is in may never
        // complete (another arrival would overrun its count), and a copy could be on its way into the stage: stop here.
        if (*reinterpret_cast<volatile int*>(&s_gave_up) != 0) break;
#pragma unroll
        for (int i = 0; i < chunks; ++i) {
          const uint32_t src = smem_u32(outs + slot * out_slot + i * out_chunk);
          const int x = rank * U + i * kRegChunk;
          if (own_dwx) tma_store_5d(&dwx_map, src, x, n, b0, 0, t0);
          tma_store_5d(&dgr_map, src + ring_steps * dwx_bytes, x, n, b0, 0, t0);
        }
        tma_store_commit();
        // A warp that stages into this slot again has read the inputs asked for below, after these copies have read the slot.
        tma_store_wait_read<0>();
        if (t0 - kRegSlots * ring_steps >= 0) fill(t0 - kRegSlots * ring_steps, slot);
        if (++slot == kRegSlots) { slot = 0; phase ^= 1u; }
      }
      tma_store_wait<0>();
    }
    __syncwarp();
  } else {
    // A fragments of R_slice^T: 8x8 blocks of R are loaded as they lie (gate rows x units p) and transposed in the warp.
    const int n_tiles = D / 16;
    // One CTA: a warp per (tile, sum) pair, the others have no product. Cluster: tiles warp, warp + 8, ... and all of their sums.
    const bool has_pair = !LOCAL || warp < (KT == 3 ? 9 : KT);
    const int source0 = LOCAL ? (KT == 3 ? warp / 3 : 0) : rank * CH;
    const int tile0 = LOCAL ? (KT == 3 ? warp % 3 : warp) : warp;
    uint32_t a[MTW][CH * KTW][4];
#pragma unroll
    for (int m = 0; m < MTW; ++m)
#pragma unroll
      for (int j = 0; j < CH * KTW; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          // first gate row (gate, unit of the CTA) of k tile j: contiguous, or gate j % GR of 16 units
          const int row = (HALVES ? j % KTW * U + j / KTW * 16 : (LOCAL && KT == 3 ? j * U + 16 * source0 : j * 16)) + 8 * (r >> 1) + q;
          const int g = row / U, u = row % U;
          const int pcol = (tile0 + nwarps * m) * 16 + 8 * (r & 1) + 2 * c;
          uint32_t v = 0u;
          if (has_pair && pcol < D && rank * U + u < D)
            v = __ldg(reinterpret_cast<const uint32_t*>(p.R + ((static_cast<size_t>(g) * N + n) * D + rank * U + u) * D + pcol));
          a[m][j][r] = movmatrix_trans(v);
        }

    const int ul = warp * UPW + (q & 3), d = rank * U + ul;
    auto item_row = [&](int i) { return i * 8 + 2 * c + hi; };  // lanes 0 - 15 have the even rows of a column tile, 16 - 31 the odd ones
    const size_t ND = static_cast<size_t>(N) * D, BND = static_cast<size_t>(B) * ND;
    const size_t sBTND = static_cast<size_t>(T) * BND;
    const bool own = !HALVES || d < D;  // false in four warps of the last CTA, which take part in the products only
    bool act[NB];
    float dcar[S][NB], dbacc[CT::GB][NB], sn[HS][NB];
#pragma unroll
    for (int g = 0; g < CT::GB; ++g)
#pragma unroll
      for (int e = 0; e < NB; ++e) dbacc[g][e] = 0.0f;
#pragma unroll
    for (int e = 0; e < NB; ++e) {
      const size_t b = static_cast<size_t>(b0 + item_row(e));
      act[e] = own && b < static_cast<size_t>(B);
#pragma unroll
      for (int k = 0; k < S; ++k) dcar[k][e] = act[e] ? p.d_carry[k * BND + b * ND + static_cast<size_t>(n) * D + d] : 0.0f;
#pragma unroll
      for (int k = 0; k < HS; ++k)
        sn[k][e] = act[e] ? history[(HP + k) * sBTND + ((b * T + T - 1) * N + n) * D + d] : 0.0f;
    }
    const int uc = ul % kRegChunk;  // unit inside the staged 32
    // offsets of the thread's item in a plane; that of the second column tile is 8 rows further
    const uint32_t off2 = reg_tile_offset<2, kRegChunk>(item_row(0), uc), off4 = reg_tile_offset<4, kRegChunk>(item_row(0), uc);
    const uint32_t my_chunk = smem_u32(stages) + ul / kRegChunk * ring_steps * Cfg::CHUNK, my_out = smem_u32(outs) + ul / kRegChunk * out_chunk;
    constexpr int compute_threads = nwarps * 32;
    const bool v1 = p.slstm_v1 != 0, zero_first = p.slstm_zero_first != 0, cut = p.cut_recurrent != 0, clip_on = p.grad_clip > 0.0f;
    const float grad_clip = p.grad_clip;
    // where this lane's words of a tile go: the rows q and q + 8 of the tile, batch rows 2c and 2c + 1
    const uint32_t row_off = smem_u32(part) + static_cast<uint32_t>(source0 * kPartSource + ((tile0 & 1) * 16 + q) * kUnit + c * 8);
    uint32_t owner_delta[MTW];  // shared memory of the CTA that owns the tile's units: 32 of them, two tiles
#pragma unroll
    for (int m = 0; m < MTW; ++m) {
      const int tile = tile0 + nwarps * m;
      owner_delta[m] = LOCAL ? static_cast<uint32_t>(tile / 2 * 32 * kUnit) : map_to_cta(smem_u32(smem), tile < n_tiles ? tile / 2 : rank) - smem_u32(smem);
    }

    bool dead = false;  // warp-uniform: after a failed wait the warp walks on without waiting
    auto give_up = [&](int code, int it) {
      if (lane == 0) reg_report(p.err, code, it);
      dead = true;
      *reinterpret_cast<volatile int*>(&s_gave_up) = 1;
    };
    if (!LOCAL) cluster_sync_all();
    if (prof) p.err[20] = static_cast<int>(clock64() - t_entry);

    constexpr int kSrc = Cfg::MAX_SOURCES < 8 ? Cfg::MAX_SOURCES : 8;  // sources read at once
    // Partial sums of iteration `it`, added to ds in the order of their sources.
    auto add_parts = [&](int it, float (&dsum)[NB]) {
      const uint32_t pbuf = smem_u32(part) + (it & 1) * part_bytes + ul * kUnit + (2 * c + hi) * 4;
#pragma unroll
      for (int k0 = 0; k0 < Cfg::MAX_SOURCES; k0 += kSrc) {
        float v[kSrc][NB];
#pragma unroll
        for (int k = 0; k < kSrc; ++k)
#pragma unroll
          for (int e = 0; e < NB; ++e) v[k][e] = k0 + k < sources ? lds_f32(pbuf + (k0 + k) * kPartSource + e * kPartTile) : 0.0f;
#pragma unroll
        for (int k = 0; k < kSrc; ++k)
#pragma unroll
          for (int e = 0; e < NB; ++e) dsum[e] += v[k][e];
      }
    };
    // The steps, compiled without the options and hooks of a call, with the options, and with both: their flags are a good part of a
    // step's instructions, and the phase timers' registers are spilled fragments elsewhere (LSTM B9 T256 N1 D512 with a clip, us: 581 in a loop
    // with the hooks, 374 without).
    auto run = [&](auto mode_tag) {
      constexpr bool hook = decltype(mode_tag)::value == kRegHooks, any = decltype(mode_tag)::value != kRegPlain;
      long long pc[6] = {0, 0, 0, 0, 0, 0};
      auto clock = [&]() -> long long { return hook && prof ? clock64() : 0; };
      // what a silenced iteration leaves out is waited for on a barrier that nobody arrives at (one CTA) or that stays incomplete
      auto wait_parts = [&](int it) {
        if constexpr (LOCAL) {
          asm volatile("bar.sync 2, %0;" ::"n"(compute_threads) : "memory");
          if (hook && it > mute_from && !dead && !mbar_wait_warp<false>(smem_u32(&s_part_bar[0]), 0, limit, abort_flag)) give_up(kErrWaitPart, it);
        } else {
          if (!dead && !mbar_wait_warp<true>(smem_u32(&s_part_bar[it & 1]), ((it - 1) >> 1) & 1, limit, abort_flag)) give_up(kErrWaitPart, it);
        }
      };
      int slot = 0, it = 0;
      uint32_t in_phase = 0;
      for (int t0 = (T - 1) / ring_steps * ring_steps; t0 >= 0; t0 -= ring_steps) {
        if (!dead && !mbar_wait_warp<false>(smem_u32(&s_full[slot]), in_phase, limit, abort_flag)) give_up(kErrWaitWx, it);
        const int first = T - 1 - it - t0;  // step of the transfer it begins with, counting down
        const uint32_t in = my_chunk + slot * stage_bytes, out = my_out + slot * out_slot;
        uint32_t in_c = in + first * (GCL * Cfg::PLANEC);
        uint32_t in_h = in + ring_steps * (GCL * Cfg::PLANEC) + first * (HS * kPlane4) + off4;
        uint32_t in_d = in + ring_steps * (GCL * Cfg::PLANEC + HS * kPlane4) + first * (S * kPlane4) + off4;
        uint32_t out_w = out + first * dwx_bytes;
        uint32_t out_g = out + ring_steps * dwx_bytes + first * (CT::GR * kPlane2) + off2;
        for (int t = t0 + first; t >= t0; --t, ++it) {
          if (hook && jitter != 0u) { jitter_stall(jitter, static_cast<uint32_t>(warp), static_cast<uint32_t>(it)); __syncwarp(); }
          const long long c1 = clock();
          float cache[CT::GC][NB], sp[HS][NB], dh[S][NB], ds[S][NB];
#pragma unroll
          for (int e = 0; e < NB; ++e) {
            const int far4 = e * (8 * kRegChunk * 4), farc = e * (8 * kRegChunk * CT::CES);
#pragma unroll
            for (int g = 0; g < GCL; ++g) {
              if constexpr (CT::CES == 2) cache[g][e] = __half2float(__ushort_as_half(static_cast<unsigned short>(lds_u16(in_c + off2 + g * Cfg::PLANEC + farc))));
              else cache[g][e] = lds_f32(in_c + off4 + g * Cfg::PLANEC + farc);
            }
#pragma unroll
            for (int k = 0; k < HS; ++k) sp[k][e] = lds_f32(in_h + k * kPlane4 + far4);
#pragma unroll
            for (int k = 0; k < S; ++k) dh[k][e] = lds_f32(in_d + k * kPlane4 + far4);
          }
          in_c -= GCL * Cfg::PLANEC;
          in_h -= HS * kPlane4;
          in_d -= S * kPlane4;
          if (t == 0) {
#pragma unroll
            for (int e = 0; e < NB; ++e)
#pragma unroll
              for (int k = 0; k < HS; ++k)
                if (act[e]) sp[k][e] = initial[(HP + k) * BND + static_cast<size_t>(b0 + item_row(e)) * ND + static_cast<size_t>(n) * D + d];
          }
#pragma unroll
          for (int k = 0; k < S; ++k)
#pragma unroll
            for (int e = 0; e < NB; ++e) ds[k][e] = dcar[k][e] + dh[k][e];
          long long cw = c1;
          if (it >= 1) {
            wait_parts(it);
            cw = clock();
            if (!(any && cut)) add_parts(it, ds[0]);
          }
          if (any && clip_on && it >= 1) {
            // the gradient carried into h_t from step t + 1 (total minus the external part) is complete here: clip it
#pragma unroll
            for (int e = 0; e < NB; ++e) ds[0][e] = clip_sym(ds[0][e] - dh[0][e], grad_clip) + dh[0][e];
          }
          if (HALVES && !own) {
#pragma unroll
            for (int e = 0; e < NB; ++e) ds[0][e] = 0.0f;  // nobody sends sums for units that do not exist
          }
          const long long c2 = clock();
          float dgr[CT::GR][NB], dgw[CT::GW][NB];
          const bool take_i = CELL == kSLSTM && t == 0 && zero_first;
#pragma unroll
          for (int e = 0; e < NB; ++e) {
            float cj[CT::GC], snj[S], spj[S], dsj[S], gr[CT::GR], gw[CT::GW], gb[CT::GB];
#pragma unroll
            for (int g = 0; g < GCL; ++g) cj[g] = cache[g][e];
#pragma unroll
            for (int k = 0; k < S; ++k) {
              snj[k] = k >= HP && k < HP + HS ? sn[k >= HP ? k - HP : 0][e] : 0.0f;
              spj[k] = k >= HP && k < HP + HS ? sp[k >= HP ? k - HP : 0][e] : 0.0f;
              dsj[k] = ds[k][e];
            }
            cell_backward<CELL>(cj, spj, snj, dsj, gr, gw, gb, take_i, any && v1);
            // Rows past the batch and units past the head hold zeros: so do their gradients, but where the cell divides.
            constexpr bool drop = CELL == kSLSTM;
#pragma unroll
            for (int k = 0; k < S; ++k) dcar[k][e] = !drop || act[e] ? dsj[k] : 0.0f;
#pragma unroll
            for (int g = 0; g < CT::GR; ++g) dgr[g][e] = !drop || act[e] ? gr[g] : 0.0f;
#pragma unroll
            for (int g = 0; g < CT::GW; ++g) dgw[g][e] = !drop || act[e] ? gw[g] : 0.0f;
          }
          uint32_t dgp[CT::GR][NB];  // bf16
          const uint32_t dgs = smem_u32(dgbuf) + (it & 1) * (NB * Cfg::DG_BYTES);
#pragma unroll
          for (int g = 0; g < CT::GR; ++g)
#pragma unroll
            for (int e = 0; e < NB; ++e) {
              dgp[g][e] = bf16_bits(dgr[g][e]);
              sts_u16(dgs + (ul * 16 + (2 * c + hi) * 2) + e * Cfg::DG_BYTES + g * U * 16, dgp[g][e]);
            }
#pragma unroll
          for (int k = 0; k < HS; ++k)
#pragma unroll
            for (int e = 0; e < NB; ++e) sn[k][e] = sp[k][e];
          asm volatile("bar.sync 1, %0;" ::"n"(compute_threads) : "memory");
          const long long c3 = clock();
          const int nb = (it + 1) & 1;
          const bool publish = !dead && !(hook && it >= mute_from);
          if (has_pair) {
            // Two column tiles: side by side where a warp has one row tile, else one after the other.
            constexpr int NP = MTW * CH == 1 ? NB : 1;
#pragma unroll
            for (int e0 = 0; e0 < NB; e0 += NP) {
              float acc[NP][CH][MTW][4];
#pragma unroll
              for (int e = 0; e < NP; ++e)
#pragma unroll
                for (int h = 0; h < CH; ++h)
#pragma unroll
                  for (int m = 0; m < MTW; ++m)
#pragma unroll
                    for (int r = 0; r < 4; ++r) acc[e][h][m][r] = 0.0f;
              // k tiles two at a time (with HALVES: gate g of both sums); the lanes 16 - 31 point at the second one's rows
              constexpr int kPair = LOCAL && KT == 3 ? 2 * U * 16 : 512;
              const uint32_t lane_off = LOCAL && KT == 3 ? static_cast<uint32_t>(((lane >> 4) * U + 16 * source0 + (lane & 15)) * 16) : lane * 16;
              constexpr int pairs = HALVES ? KTW : KTW / 2;
#pragma unroll
              for (int k2 = 0; k2 < pairs; ++k2) {
#pragma unroll
                for (int e = 0; e < NP; ++e) {
                  uint32_t bf[4];
                  ldsm_x4_trans(dgs + lane_off + (e0 + e) * Cfg::DG_BYTES + k2 * kPair, bf);
#pragma unroll
                  for (int m = 0; m < MTW; ++m) mma_bf16_16816(acc[e][0][m], a[m][HALVES ? k2 : 2 * k2], bf[0], bf[1]);
#pragma unroll
                  for (int m = 0; m < MTW; ++m) mma_bf16_16816(acc[e][CH - 1][m], a[m][HALVES ? KTW + k2 : 2 * k2 + 1], bf[2], bf[3]);
                }
              }
              if constexpr (!HALVES && KTW % 2 == 1) {
#pragma unroll
                for (int e = 0; e < NP; ++e) {
                  uint32_t b0w, b1w;
                  ldsm_x2_trans(dgs + (e0 + e) * Cfg::DG_BYTES + (LOCAL && KT == 3 ? ((KTW - 1) * U + 16 * source0) * 16 : (KTW - 1) * 256) + (lane & 15) * 16, b0w, b1w);
#pragma unroll
                  for (int m = 0; m < MTW; ++m) mma_bf16_16816(acc[e][0][m], a[m][KTW - 1], b0w, b1w);
                }
              }
#pragma unroll
              for (int e = 0; e < NP; ++e)
#pragma unroll
                for (int h = 0; h < CH; ++h)
#pragma unroll
                  for (int m = 0; m < MTW; ++m) {
                    const float(&v)[4] = acc[e][h][m];
                    const uint32_t dst = row_off + owner_delta[m] + nb * part_bytes + h * kPartSource + (e0 + e) * kPartTile;
                    if constexpr (LOCAL) {
                      if (publish) {
                        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(dst), "f"(v[0]), "f"(v[1]) : "memory");
                        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(dst + 8 * kUnit), "f"(v[2]), "f"(v[3]) : "memory");
                      }
                    } else {
                      const uint32_t bar = smem_u32(&s_part_bar[nb]) + owner_delta[m];
                      if (publish && tile0 + nwarps * m < n_tiles && (!HALVES || source0 + h < sources)) {
                        st_async_v2_b32(dst, __float_as_uint(v[0]), __float_as_uint(v[1]), bar);
                        st_async_v2_b32(dst + 8 * kUnit, __float_as_uint(v[2]), __float_as_uint(v[3]), bar);
                      }
                    }
                  }
            }
          }
          const long long c4 = clock();
          // outputs, while the partial sums of the next step are on their way
#pragma unroll
          for (int e = 0; e < NB; ++e)
#pragma unroll
            for (int g = 0; g < CT::GR; ++g) sts_u16(out_g + g * kPlane2 + e * (8 * kRegChunk * 2), dgp[g][e]);
          if (own_dwx) {
#pragma unroll
            for (int e = 0; e < NB; ++e)
#pragma unroll
              for (int g = 0; g < CT::GW; ++g) {
                if (wx_bf16) sts_u16(out_w + off2 + g * kPlane2 + e * (8 * kRegChunk * 2), bf16_bits(dgw[g][e]));
                else sts_f32(out_w + off4 + g * kPlane4 + e * (8 * kRegChunk * 4), dgw[g][e]);
              }
          }
          out_w -= dwx_bytes;
          out_g -= CT::GR * kPlane2;
          // this parity's partial sums were complete at the wait above: armed for iteration it + 2
          if (!LOCAL && tid == 0 && !dead && it >= 1 && it + 2 <= T) mbar_arrive_expect_tx(smem_u32(&s_part_bar[it & 1]), part_tx);
#pragma unroll
          for (int g = 0; g < CT::GB; ++g)
#pragma unroll
            for (int e = 0; e < NB; ++e) dbacc[g][e] += CELL != kGRU ? dgw[g][e] : (g == 0 ? dgr[0][e] : dgw[g > 0 ? g - 1 : 0][e]);  // as cell_backward's gb
          const long long c5 = clock();
          if (hook && prof) {
            pc[0] += c5 - c1; pc[1] += c2 - c1; pc[2] += c3 - c2; pc[3] += c5 - c4; pc[4] += c4 - c3; pc[5] += cw - c1;
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&s_out_full[slot]));
        if (++slot == kRegSlots) { slot = 0; in_phase ^= 1u; }
      }
      wait_parts(T);
      if (!(any && cut)) add_parts(T, dcar[0]);
      if (hook && prof) {  // the slots of the tcgen05 kernels' phase timers that have a counterpart here
        p.err[15] = static_cast<int>(pc[0]);  // the whole step
        p.err[9] = static_cast<int>(pc[1]);   // tiles read, wait for the partial sums, their sum
        p.err[10] = static_cast<int>(pc[2]);  // cell, dg to shared memory, CTA barrier
        p.err[11] = static_cast<int>(pc[3]);  // outputs staged
        p.err[12] = static_cast<int>(pc[4]);  // mma and scatter
        p.err[13] = static_cast<int>(pc[5]);  // tiles read, wait
      }
    };
    // The options have kernels of their own, but naming them here keeps the plain loop's schedule: GRU B16 T1024 N24 D32 455 us against 459,
    // LSTM B8 T96 N48 D16 27.8 against 28.9.
    if (hooks || (!EXTRA && (cut || clip_on || v1))) run(std::integral_constant<int, kRegHooks>{});
    else run(std::integral_constant<int, EXTRA ? kRegAny : kRegPlain>{});
#pragma unroll
    for (int e = 0; e < NB; ++e)
      if (act[e]) {
#pragma unroll
        for (int k = 0; k < S; ++k)
          p.d_initial[k * BND + static_cast<size_t>(b0 + item_row(e)) * ND + static_cast<size_t>(n) * D + d] = dcar[k][e];
      }
    // bias gradient of the batch rows of the group, added in their order; an entry of db_part stands for db_rows of them
#pragma unroll
    for (int g = 0; g < CT::GB; ++g) {
      float v = 0.0f;
#pragma unroll
      for (int e = 0; e < NB; ++e) {
        if (e > 0 && (NB == 3 || p.db_rows == kRegRows)) v = 0.0f;
#pragma unroll
        for (int k = 0; k < kRegRows; ++k) v += __shfl_sync(0xffffffffu, dbacc[g][e], (k & 1) * 16 + (lane & 12) + (k >> 1));
        const int b = b0 + e * kRegRows;
        if (c == 0 && hi == 0 && own && b < B) {
          float* dst = p.db_part + ((static_cast<size_t>(b / p.db_rows) * CT::GB + g) * N + n) * D + d;
          // The halves of a 16-row entry may come from two groups: at most two addends on top of the launcher's zeros, so the order
          // cannot matter, but the sum may differ in its last bits from the 16 rows added one by one.
          if (NB != 2 && p.db_rows != kRegRows) atomicAdd(dst, v);
          else *dst = v;
        }
      }
    }
  }
  if (*abort_flag != 0) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  __syncthreads();
  if (!LOCAL) cluster_sync_all();
}

// Runs the call, or (ask) only says whether it would: kRegTaken / kRegNoRoom.
template <int CELL, int KT, bool LOCAL, bool HALVES, int NB, bool DENSE = false>
int launch_bwd_reg(const BwdParams& p, const void* cache, const float* history, const float* initial,
                   const float* d_history, int wx_bf16, cudaStream_t stream, bool ask, long long rival_groups = 0) {
  using Cfg = BwdRegCfg<CELL, KT, LOCAL, HALVES, NB, DENSE>;
  using CT = CellTraits<CELL>;
  constexpr int U = Cfg::U, ROWS = Cfg::ROWS, chunks = (U + kRegChunk - 1) / kRegChunk;
  const int C = (p.D + U - 1) / U;
  // cells whose W-gates are their R-gates may have one bf16 buffer for dWx and dg
  const bool own_dwx = !wx_bf16 || CELL == kGRU || p.dwx != static_cast<void*>(p.dgr);
  const int out_step = ROWS * kRegChunk * (CT::GR * 2 + (own_dwx ? CT::GW * (wx_bf16 ? 2 : 4) : 0));
  const int fixed = Cfg::DG_ALL + 2 * (LOCAL ? Cfg::MAX_SOURCES : (HALVES ? p.D / 16 : C)) * U * ROWS * 4;
  const int steps = reg_transfer_steps(fixed, chunks * (Cfg::CHUNK + out_step), Cfg::MIN_BLOCKS);
  const int smem = fixed + kRegSlots * chunks * (steps * Cfg::CHUNK + reg_round_1k(steps * out_step));
  if (smem > kRegSmemLimit) return kRegNoRoom;
  const int D = p.D, N = p.N, B = p.B;
  const uint64_t nd = static_cast<uint64_t>(N) * D, uT = p.T, uB = p.B;
  // bulk stores start on 16-byte boundaries; the tcgen05 kernels write these outputs with plain stores
  if (((reinterpret_cast<uintptr_t>(p.dwx) | reinterpret_cast<uintptr_t>(p.dgr)) & 15u) != 0) return kRegNoRoom;
  auto kern = reg_extra(p) ? frnn_bwd_reg_kernel<CELL, KT, LOCAL, HALVES, NB, DENSE, true> : frnn_bwd_reg_kernel<CELL, KT, LOCAL, HALVES, NB, DENSE, false>;
  BwdParams q = p;
  q.C = C;
  const long long groups = static_cast<long long>(N) * reg_batch_tiles(B, ROWS);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(groups * C));
  cfg.blockDim = dim3(static_cast<unsigned>(Cfg::THREADS));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(C);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = LOCAL ? 0 : 1;
  if constexpr (LOCAL && KT == 2 && NB == 1 && !DENSE && (CELL == kLSTM || CELL == kSLSTM)) {
    // Heads of 32 units have 288 threads: two CTAs an SM within 96 registers, three within 72 and some spills, which are a seventh (LSTM) to a
    // third (sLSTM) of a step. B304 T48 N8 (three fit, two do not), us: LSTM 52 against 59 with 16 rows, sLSTM 76 / 84; B600 89 / 105 and 142 / 167.
    const int two = reg_capacity(reinterpret_cast<const void*>(kern), cfg, 1), three = two / 2 * 3;
    const long long waves = two > 0 ? (groups + two - 1) / two : 0, dense = three > 0 ? (groups + three - 1) / three : 0;
    if (20 * waves > (CELL == kLSTM ? 23 : 27) * dense)
      return launch_bwd_reg<CELL, KT, LOCAL, HALVES, NB, true>(p, cache, history, initial, d_history, wx_bf16, stream, ask, rival_groups);
  }
  // whether the call is taken at all comes first: one that is not pays for nothing else
  const int rc = reg_room(reinterpret_cast<const void*>(kern), cfg, C, groups, rival_groups, D);
  if (rc != 0 || ask) return rc != 0 ? rc : kRegTaken;
  CUtensorMap cache_map, hist_map, dhist_map, dgr_map, dwx_map;
  const auto map = [&](CUtensorMap* m, const void* base, int es, int planes, int steps_end, uint64_t bs, uint64_t ps, uint64_t ss, int box_planes) {
    return reg_tile_map(m, base, es, D, N, B, planes, steps_end, bs, ps, ss, box_planes, kRegChunk, ROWS, steps);
  };
  if (map(&hist_map, history, 4, CT::S, p.T, uT * nd, uB * uT * nd, nd, Cfg::HS) != 0 ||
      map(&dhist_map, d_history, 4, CT::S, p.T, uT * nd, uB * uT * nd, nd, CT::S) != 0 ||
      map(&dgr_map, p.dgr, 2, CT::GR, p.T, uT * CT::GR * nd, nd, CT::GR * nd, CT::GR) != 0)
    return -4;
  cache_map = hist_map;  // Elman has no cache: a valid map that is never used
  if (Cfg::GCL > 0 && map(&cache_map, cache, CT::CES, CT::GC, p.T, uT * CT::GC * nd, nd, CT::GC * nd, CT::GC) != 0) return -4;
  dwx_map = dgr_map;
  if (own_dwx && map(&dwx_map, p.dwx, wx_bf16 ? 2 : 4, CT::GW, p.T, uT * CT::GW * nd, nd, CT::GW * nd, CT::GW) != 0) return -4;
  if (NB != 2 && p.db_rows != kRegRows) {
    const size_t tiles = static_cast<size_t>((p.B + p.db_rows - 1) / p.db_rows);
    const cudaError_t e = cudaMemsetAsync(p.db_part, 0, tiles * CT::GB * p.N * p.D * sizeof(float), stream);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, q, history, initial, cache_map, hist_map, dhist_map, dgr_map, dwx_map,
                                             wx_bf16, own_dwx ? 1 : 0, steps));
}

struct BwdRegCall {
  const BwdParams& p;
  const void* cache;
  const float *history, *initial, *d_history;
  int wx_bf16;
  cudaStream_t stream;
  int rows;
  bool ask;
};

template <int CELL, int KT, bool LOCAL, bool HALVES>
int launch_bwd_reg_rows(const BwdRegCall& v) {
  const long long rivals = LOCAL ? static_cast<long long>(v.p.N) * reg_batch_tiles(v.p.B, 16) : 0;
  if (v.rows == kRegRows)
    return launch_bwd_reg<CELL, KT, LOCAL, HALVES, 1>(v.p, v.cache, v.history, v.initial, v.d_history, v.wx_bf16, v.stream, v.ask, rivals);
  // Where registers run out (the sLSTM from 288 units on and with two sums a tile, four gates beyond 384 units), or the tcgen05 kernel's
  // clusters of 9 still run two to an SM, more rows per group are no faster than that kernel. T48 N1 - 4, us, against it: 16 rows sLSTM B64
  // D320 127 / 157, D288 126 / 120, D448 322 / 253, B256 D112 177 / 168; 24 rows LSTM B64 D384 162 / 245, B256 D288 160 / 149, B56
  // D512 (T64) 400 / 354; GRU B256 D288 95 / 131.
  // 16 rows of an LSTM from 448 units on with fp32 Wx (a second output to stage) win by the second wave that the tcgen05 groups need, and
  // lose against a single one: D512 189 / 213 and 193 / 145. tcgen05 groups of 8 rows (db_rows: few groups) beat 24 rows of four gates, LSTM B22
  // N4 D384 146 / 105.
  constexpr bool tight = CELL == kLSTM || CELL == kSLSTM;
  const bool few = v.p.db_rows == kRegRows;
  if (v.rows == 2 * kRegRows) {
    if ((CELL == kSLSTM && (HALVES || KT == 32 || v.p.D == 288))) return kRegNoRoom;
    if (CELL == kLSTM && v.p.D >= 448 && !v.wx_bf16 && reg_rival(true, CELL, v.wx_bf16, v.p.N, v.p.B, v.p.D).waves == 1) return kRegNoRoom;
    return launch_bwd_reg<CELL, KT, LOCAL, HALVES, 2>(v.p, v.cache, v.history, v.initial, v.d_history, v.wx_bf16, v.stream, v.ask, rivals);
  }
  if constexpr (KT >= 16 && !HALVES && !(tight && KT == 32)) {
    if (tight && (v.p.D == 288 || few)) return kRegNoRoom;
    return launch_bwd_reg<CELL, KT, LOCAL, HALVES, 3>(v.p, v.cache, v.history, v.initial, v.d_history, v.wx_bf16, v.stream, v.ask);
  }
  return kRegNoRoom;
}

template <int CELL, int KT>
int launch_bwd_reg_cluster(const BwdRegCall& v) {
  if (v.p.D % 32 != 0) {
    // The odd multiples of 16 begin at 80. The sLSTM at 208 and 240 units needs all 255 registers and is no faster here than
    // on the tcgen05 kernel: T128 N1, forward and backward, 399 us against 378 at B4 D208 and 488 against 478 at B48 D240.
    if constexpr (KT > 4 && KT <= 16) return CELL == kSLSTM && v.p.D > 192 ? kRegNoRoom : launch_bwd_reg_rows<CELL, KT, false, true>(v);
    else return kRegNoRoom;
  }
  return launch_bwd_reg_rows<CELL, KT, false, false>(v);
}

}  // namespace

template <int CELL>
int launch_bwd_reg_cell(const BwdParams& p, const void* cache, const float* history, const float* initial,
                        const float* d_history, int wx_bf16, cudaStream_t s, int rows, bool ask) {
  const BwdRegCall v{p, cache, history, initial, d_history, wx_bf16, s, rows, ask};
  switch (reg_k_tiles(p.D)) {  // in a cluster KT only bounds the row tiles of a warp and the sources
    case 1: return launch_bwd_reg_rows<CELL, 1, true, false>(v);
    case 2: return launch_bwd_reg_rows<CELL, 2, true, false>(v);
    case 3: return launch_bwd_reg_rows<CELL, 3, true, false>(v);
    case 4: return launch_bwd_reg_cluster<CELL, 4>(v);
    case 6:
    case 8: return launch_bwd_reg_cluster<CELL, 8>(v);
    case 10:
    case 12:
    case 14:
    case 16: return launch_bwd_reg_cluster<CELL, 16>(v);
    case 20:
    case 24: return launch_bwd_reg_cluster<CELL, 24>(v);
    case 28:
    case 32: return launch_bwd_reg_cluster<CELL, 32>(v);
    default: return -2;
  }
}

}  // namespace frnn
