// Forward recurrence of heads of 576 to 1024 units with R in the register file (see recurrent_reg.cuh, recurrent_reg_fwd.cuh).
//
// The decomposition is that of recurrent_fwd_ksplit.cu: a group (head, 8 or 16 batch rows) is D/32 row tiles of 32 units times KS
// chunks of the contraction, the KS CTAs of a tile are a cluster. Warp w of a CTA has the fragments of units 4w .. 4w + 3 of the
// tile, all gates, for its chunk. Per step
//   1. every warp multiplies its fragments with the chunk of round_bf16(h_{t-1}) in shared memory and sends the partial gates of an
//      item (unit, batch row), 16 bytes, to the CTA that owns the unit (32 / KS units each; st.async),
//   2. the owner warps add the KS partial sums in their order (the sums are those of the tensor-memory kernel, bit for bit), run the
//      cell and store the words of h_t (two batch rows of a unit) to the group's slot of the step in global memory,
//   3. all warps fetch the packets (8 batch rows of a unit) of their chunk: a packet whose words all differ from the fill has arrived.
//
// Slots: kWideSlots of them in turn, filled with ones by the caller. The slot that a step writes was refilled kWideSlots / 2 steps
// before, by the lanes that have no data to store; it had been read kWideSlots / 2 steps before that. Every kWideFence steps each thread
// fences: the refill of step t is ordered (by the barrier of a step) before a fence of its CTA at step t + kWideFence at the
// latest, that one before the data of the step after it, whose reader fences by step t + 2 * kWideFence + 1, long before it polls the
// refilled slot at step t + kWideSlots / 2. So no reader can take old data of a slot for new.
//
// Bound: the serial chain of a step, two hops of it: LSTM B16 N1 D768 (KS = 2), cycles: h_t of the other CTAs polled 1075, ldmatrix, mma
// and partial gates sent 755, wait for the partial gates and their sum 583, cell and publication 227, staging 224. us per step of the
// tensor-memory kernel and here: there 2.31 / 1.73, B4 (KS = 4) 2.12 / 1.62; D1024 B8 2.35 / 1.71. What went: tcgen05.mma, its commit and
// tcgen05.ld (950 cycles against 300 of mma.sync), a fence per step (now one in kWideFence), scattered output stores.
#pragma once

#include <algorithm>
#include <type_traits>

#include "recurrent_reg.cuh"

namespace frnn {

namespace {

template <int CELL, int KS, int NB, int KT>
struct FwdWideCfg {
  using CT = CellTraits<CELL>;
  static constexpr int UO = 32 / KS, OWNERS = UO * NB / 4;          // units owned, warps that run their cells
  static constexpr int ROWS = NB * kRegRows, CHUNK = UO, THREADS = 9 * 32;
  static constexpr int PACKET = CT::GR == 1 ? 4 : 16;              // partial gates of an item
  static constexpr int HALF = KT * 256, HBUF = NB * HALF;          // operand: [column tile][k][8 batch rows]
  static constexpr int PART = KS * NB * UO * 8 * PACKET;           // one parity: [source][column tile][unit][batch row]
  static constexpr int FIXED = reg_round_1k(2 * HBUF + 2 * PART);
  static_assert(OWNERS <= 8, "an item per thread");
};

template <int CELL, int KS, int NB, int KT, bool EXTRA>
__global__ void __launch_bounds__(FwdWideCfg<CELL, KS, NB, KT>::THREADS, 1)
frnn_fwd_wide_kernel(const FwdParams p, const __grid_constant__ CUtensorMap wx_map, const __grid_constant__ CUtensorMap hist_map,
                     const __grid_constant__ CUtensorMap cache_map, const __grid_constant__ CUtensorMap hbf_map, const int wx_bf16,
                     const int ring_steps, const int hist_states, const int xg_slots) {
  using Cfg = FwdWideCfg<CELL, KS, NB, KT>;
  using CT = CellTraits<CELL>;
  constexpr int UO = Cfg::UO, CHUNK = Cfg::CHUNK, ROWS = Cfg::ROWS, OWNERS = Cfg::OWNERS, PACKET = Cfg::PACKET;
  constexpr int kPlane2 = ROWS * CHUNK * 2, kPlane4 = ROWS * CHUNK * 4, kPlaneC = ROWS * CHUNK * CT::CES;

  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t s_part_bar[2];
  __shared__ int s_gave_up;  // a compute warp of this CTA has stopped waiting
  __shared__ __align__(8) uint64_t s_out_full[kRegSlots];
  __shared__ __align__(8) uint64_t s_wx_full[kRegSlots];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane >> 2, c = lane & 3, hi = lane >> 4, uq = q & 3;
  const long long t_entry = clock64();
  const int D = p.D, N = p.N, T = p.T, B = p.B, RT = D / 32, Kc = D / KS;
  const int ks = static_cast<int>(blockIdx.x % KS);  // == rank inside the cluster
  const int rt = static_cast<int>(blockIdx.x / KS % RT), gid = static_cast<int>(blockIdx.x / (KS * RT));
  const int n = gid % N, b0 = gid / N * ROWS;
  uint8_t* const hbuf = smem;
  uint8_t* const part = smem + 2 * Cfg::HBUF;
  uint8_t* const wxs = smem + Cfg::FIXED;
  const int step_in = CT::GW * (wx_bf16 ? kPlane2 : kPlane4), stage_bytes = reg_round_1k(ring_steps * step_in);
  const bool out_bf16 = p.out_bf16 != 0, has_cache = p.cache != nullptr && CELL != kElman, has_hbf = p.hbf != nullptr;
  const int hist_bytes = hist_states * (out_bf16 ? kPlane2 : kPlane4);
  const int cache_bytes = has_cache ? CT::GC * kPlaneC : 0;
  // regions of a transfer of outputs, each from a multiple of 1 KB (the swizzles follow address bits)
  const int region_c = reg_round_1k(ring_steps * hist_bytes), region_b = region_c + reg_round_1k(ring_steps * cache_bytes);
  const int out_slot = region_b + (has_hbf ? reg_round_1k(ring_steps * kPlane2) : 0);
  uint8_t* const outs = wxs + kRegSlots * stage_bytes;
  uint8_t* const xg = p.xg_data + static_cast<size_t>(gid) * xg_slots * (static_cast<size_t>(ROWS) * D * 2);
  const uint32_t slot_bytes = static_cast<uint32_t>(ROWS) * D * 2u;
  const volatile int* abort_flag = p.err;
  const uint64_t limit = p.wait_limit_ns;
  const bool zero_first = p.zero_first_dev != nullptr ? *p.zero_first_dev != 0 : p.slstm_zero_first != 0;
  // hooks of the caller: phase timers; nobody publishes from a step on; delays (fp32 Wx: see jitter_stall)
  const bool prof = p.err[3] != 0 && blockIdx.x == 0 && tid == 0;
  const int mute_from = p.err[4] != 0 ? p.err[5] : 0x7fffffff;
  const uint32_t jitter = wx_bf16 ? 0u : static_cast<uint32_t>(p.err[6]);
  const bool hooks = p.err[3] != 0 || p.err[4] != 0 || (jitter != 0u && p.err[7] == 0);  // err[7]: only the I/O warp is late

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&s_part_bar[i]), 1);
    for (int i = 0; i < kRegSlots; ++i) {
      mbar_init(smem_u32(&s_out_full[i]), OWNERS);
      mbar_init(smem_u32(&s_wx_full[i]), 1);
    }
    s_gave_up = 0;
    fence_mbar_init();
    tma_prefetch_desc(&wx_map);
  }
  // operand buffer 0 = round_bf16(initial h) of the chunk, zero for rows past the batch and k past the chunk; buffer 1 zero
  reg_fill_operand<NB, KT>(hbuf, p.initial + static_cast<size_t>(n) * D + ks * Kc, static_cast<size_t>(N) * D, b0, B, Kc, tid, blockDim.x);
  __syncthreads();
  if (tid == 0) {
    mbar_arrive_expect_tx(smem_u32(&s_part_bar[0]), Cfg::PART);
    if (T >= 2) mbar_arrive_expect_tx(smem_u32(&s_part_bar[1]), Cfg::PART);
  }

  if (warp == 8) {
    // ---------------- I/O warp: Wx tiles in, staged outputs out ----------------
    cluster_sync_all();
    if (lane == 0) {
      const int x = rt * 32 + ks * UO;
      auto fill = [&](int t, int s) {  // the inputs of the steps t .. t + ring_steps - 1
        const uint32_t bar = smem_u32(&s_wx_full[s]);
        mbar_arrive_expect_tx(bar, ring_steps * step_in);
        tma_load_5d(smem_u32(wxs + s * stage_bytes), &wx_map, bar, x, n, b0, 0, p.t0 + t);
      };
      for (int i = 0; i < kRegSlots && i * ring_steps < T; ++i) fill(i * ring_steps, i);
      int slot = 0;
      uint32_t phase = 0;
      auto staged = [&](int step) -> bool {  // as in recurrent_reg_fwd.cuh
        const uint32_t bar = smem_u32(&s_out_full[slot]);
        for (int fast = 0; fast < 64; ++fast)
          if (mbar_try_wait(bar, phase)) return true;
        if (jitter != 0u) jitter_stall(jitter, 32u, static_cast<uint32_t>(step));
        return mbar_wait_bounded<false>(bar, phase, 2 * limit, abort_flag);
      };
      for (int t = 0; t < T; t += ring_steps) {
        if (!staged(t)) {
          reg_report(p.err, kErrWaitEpi, t);
          break;
        }
        // A warp that gave up on a wait sets the flag before it stages: see recurrent_reg_fwd.cuh.
        if (*reinterpret_cast<volatile int*>(&s_gave_up) != 0) break;
        const uint32_t src = smem_u32(outs + slot * out_slot);
        if (hist_states > 0) tma_store_5d(&hist_map, src, x, n, b0, 0, p.t0 + t);
        if (has_cache) tma_store_5d(&cache_map, src + region_c, x, n, b0, 0, t);
        if (has_hbf) tma_store_5d(&hbf_map, src + region_b, x, n, b0, 0, t);
        tma_store_commit();
        // A warp that stages into this slot again has read the inputs asked for below, after these copies have read the slot.
        tma_store_wait_read<0>();
        if (t + kRegSlots * ring_steps < T) fill(t + kRegSlots * ring_steps, slot);
        if (++slot == kRegSlots) { slot = 0; phase ^= 1u; }
      }
      tma_store_wait<0>();
    }
    __syncwarp();
  } else {
    uint32_t a[KT][4];
    // the ring is scratch until the cluster has met
    reg_load_rows<KT, 4, CT::GR>(p.R + (static_cast<size_t>(n) * D + rt * 32 + warp * 4) * D + ks * Kc, static_cast<size_t>(N) * D * D, D, Kc,
                                 smem_u32(wxs) + warp * kRegScratch, lane, (reinterpret_cast<uintptr_t>(p.R) & 15u) == 0, a);

    // the item of a thread of an owner warp: one unit of one batch row
    const size_t ND = static_cast<size_t>(N) * D;
    const bool owner = warp < OWNERS;
    const int tile = warp / (UO / 4), ul = warp % (UO / 4) * 4 + uq, row = 2 * c + hi;  // column tile, unit, row of the tile
    const int d = rt * 32 + ks * UO + ul, b = b0 + tile * 8 + row;
    const bool act = owner && b < B;
    const size_t item = static_cast<size_t>(b) * ND + static_cast<size_t>(n) * D + d;
    float st[CT::S], bias[CT::GB];
#pragma unroll
    for (int g = 0; g < CT::GB; ++g) bias[g] = owner ? p.bias[(static_cast<size_t>(g) * N + n) * D + d] : 0.0f;
#pragma unroll
    for (int s = 0; s < CT::S; ++s) st[s] = act ? p.initial[static_cast<size_t>(s) * B * ND + item] : 0.0f;
    if (act && has_hbf) p.hbf[(static_cast<size_t>(b) * (T + 1)) * ND + static_cast<size_t>(n) * D + d] = __float2bfloat16_rn(st[0]);
    const bool clip_on = p.fwd_clip < INFINITY;
    const float clip = p.fwd_clip;
    const uint32_t off2 = reg_tile_offset<2, CHUNK>(tile * 8 + row, ul), off4 = reg_tile_offset<4, CHUNK>(tile * 8 + row, ul);
    // where the partial gates of this warp's units go
    const uint32_t to = static_cast<uint32_t>(4 * warp / UO);
    const uint32_t delta = map_to_cta(smem_u32(smem), to) - smem_u32(smem);
    const uint32_t part_dst = smem_u32(part) + static_cast<uint32_t>((ks * NB * UO + 4 * warp % UO + uq) * 8 + row) * PACKET;
    const uint32_t part_src = smem_u32(part) + static_cast<uint32_t>((tile * UO + ul) * 8 + row) * PACKET;
    // the word this thread stores: data for the lanes 0 - 15, the refill of a later step's slot for the lanes 16 - 31
    const uint32_t word_at = static_cast<uint32_t>(tile * D + d) * 16 + c * 4;
    // the packets this thread fetches
    constexpr int J = (NB * KT * 16 + 255) / 256;
    const int packets = NB * Kc;
    bool dead = false;  // warp-uniform: after a failed wait the warp walks on without waiting
    auto give_up = [&](int code, int t) {
      if (lane == 0) reg_report(p.err, code, t);
      dead = true;
      *reinterpret_cast<volatile int*>(&s_gave_up) = 1;
    };
    cluster_sync_all();
    if (prof) p.err[20] = static_cast<int>(clock64() - t_entry);

    // The steps, compiled for what the call writes, and for anything (with the hooks): see recurrent_reg_fwd.cuh.
    auto run = [&](auto mode_tag) {
      constexpr int MODE = decltype(mode_tag)::value;
      constexpr bool hook = MODE == kRegHooks, any = hook || MODE == kRegAny, train = MODE == kRegTrain || MODE == kRegClipped;
      const bool save = any ? has_cache : train && CELL != kElman, keep_h = any ? has_hbf : train;
      const bool narrow = any ? out_bf16 : MODE == kRegNarrow, clipped = any ? clip_on : MODE == kRegClipped;
      const int states = any || MODE == kRegNarrow ? hist_states : (MODE == kRegHidden ? 1 : (MODE == kRegLast ? 0 : CT::S));
      const int hist_step = any || MODE == kRegNarrow ? hist_bytes : states * kPlane4, cache_step = any ? cache_bytes : (save ? CT::GC * kPlaneC : 0);
      long long pc[6] = {0, 0, 0, 0, 0, 0};
      auto clock = [&]() -> long long { return hook && prof ? clock64() : 0; };
      int slot = 0;
      uint32_t in_phase = 0;
      for (int t0 = 0; t0 < T; t0 += ring_steps) {
        if (owner && !dead && !mbar_wait_warp<false>(smem_u32(&s_wx_full[slot]), in_phase, limit, abort_flag)) give_up(kErrWaitWx, t0);
        const int t_end = min(T, t0 + ring_steps);
        uint32_t in = smem_u32(wxs) + slot * stage_bytes, out_h = smem_u32(outs) + slot * out_slot;
        uint32_t out_c = out_h + region_c, out_b = out_h + region_b;
        for (int t = t0; t < t_end; ++t) {
          if (hook && jitter != 0u) { jitter_stall(jitter, static_cast<uint32_t>(warp), static_cast<uint32_t>(t)); __syncwarp(); }
          const int pb = t & 1;
          const long long c1 = clock();
          const uint32_t hb = smem_u32(hbuf) + pb * Cfg::HBUF + lane * 16;
          // One chain over the chunk's k per tile, in the order of the tensor-memory kernel.
          float acc[NB][4];
#pragma unroll
          for (int j = 0; j < NB; ++j)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[j][r] = 0.0f;
#pragma unroll
          for (int k2 = 0; k2 < KT / 2; ++k2) {
            uint32_t bf[NB][4];
#pragma unroll
            for (int j = 0; j < NB; ++j) ldsm_x4_trans(hb + j * Cfg::HALF + k2 * 512, bf[j]);
#pragma unroll
            for (int j = 0; j < NB; ++j) mma_bf16_16816(acc[j], a[2 * k2], bf[j][0], bf[j][1]);
#pragma unroll
            for (int j = 0; j < NB; ++j) mma_bf16_16816(acc[j], a[2 * k2 + 1], bf[j][2], bf[j][3]);
          }
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            const float x0 = __shfl_xor_sync(0xffffffffu, hi ? acc[j][0] : acc[j][1], 16);
            const float x1 = __shfl_xor_sync(0xffffffffu, hi ? acc[j][2] : acc[j][3], 16);
            const float g0 = hi ? x0 : acc[j][0], g1 = hi ? acc[j][1] : x0, g2 = hi ? x1 : acc[j][2], g3 = hi ? acc[j][3] : x1;
            const uint32_t dst = part_dst + delta + pb * Cfg::PART + j * (UO * 8 * PACKET), bar = smem_u32(&s_part_bar[pb]) + delta;
            if (!dead) {
              if constexpr (CT::GR == 1) st_async_b32(dst, __float_as_uint(g0), bar);
              else st_async_v4_b32(dst, __float_as_uint(g0), __float_as_uint(g1), __float_as_uint(g2), __float_as_uint(g3), bar);
            }
          }
          const long long c2 = clock();
          long long c3 = c2, c4 = c2;
          if (owner) {
            float wx[CT::GW];
#pragma unroll
            for (int g = 0; g < CT::GW; ++g)
              wx[g] = wx_bf16 ? __uint_as_float(lds_u16(in + off2 + g * kPlane2) << 16) : lds_f32(in + off4 + g * kPlane4);
            in += step_in;
            if (!dead && !mbar_wait_warp<true>(smem_u32(&s_part_bar[pb]), (t >> 1) & 1, limit, abort_flag)) give_up(kErrWaitPart, t);
            float ry[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int s = 0; s < KS; ++s) {
              const uint32_t at = part_src + pb * Cfg::PART + s * (NB * UO * 8 * PACKET);
              float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
              if constexpr (CT::GR == 1) v[0] = lds_f32(at);
              else asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(at));
#pragma unroll
              for (int g = 0; g < CT::GR; ++g) ry[g] += v[g];
            }
            c3 = clock();
            float cv[CT::GC];
            const bool take_i = CELL == kSLSTM && p.t0 + t == 0 && zero_first;
            cell_forward<CELL>(ry, wx, bias, st, cv, take_i);
            if (clipped) st[0] = fminf(fmaxf(st[0], -clip), clip);
            const float mine = act ? st[0] : 0.0f, other = __shfl_xor_sync(0xffffffffu, mine, 16);
            const bool publish = t + 1 < T && !(hook && (dead || t >= mute_from));
            if (publish && !dead) {
              const uint32_t w = hi ? kXgFill : xg_clean(pack_bf16x2(mine, other));
              const int ahead = t + 1 + (hi ? kWideSlots / 2 : 0);
              if (!hi || (ahead < T && ahead >= xg_slots))
                st_relaxed_gpu_u32(xg + static_cast<size_t>(ahead % kWideSlots) * slot_bytes + word_at, w);
            }
            c4 = clock();
            // outputs, while h_t is on its way
#pragma unroll
            for (int k = 0; k < CT::S; ++k)
              if (k < states) {
                if (narrow) sts_u16(out_h + off2 + k * kPlane2, bf16_bits(st[k]));
                else sts_f32(out_h + off4 + k * kPlane4, st[k]);
              }
            if (save) {
#pragma unroll
              for (int k = 0; k < CT::GC; ++k) {
                if constexpr (CT::CES == 2) sts_u16(out_c + off2 + k * kPlane2, __half_as_ushort(__float2half_rn(cv[k])));
                else sts_f32(out_c + off4 + k * kPlane4, cv[k]);
              }
            }
            if (keep_h) sts_u16(out_b + off2, bf16_bits(st[0]));
            out_h += hist_step;
            out_c += cache_step;
            out_b += kPlane2;
            // the barrier of this parity, complete since the wait above, is armed for step t + 2
            if (tid == 0 && !dead && t + 2 < T) mbar_arrive_expect_tx(smem_u32(&s_part_bar[pb]), Cfg::PART);
          }
          const long long c5 = clock();
          if (t + 1 < T) {
            // this CTA's chunk of h_t -> operand buffer of the next step
            const uint8_t* const from = xg + static_cast<size_t>((t + 1) % kWideSlots) * slot_bytes;
            const uint32_t dst = smem_u32(hbuf) + (pb ^ 1) * Cfg::HBUF;
            uint32_t pend = 0;
#pragma unroll
            for (int j = 0; j < J; ++j)
              if (!dead && tid + j * 256 < packets) pend |= 1u << j;
            uint64_t since = 0;
            uint32_t rounds = 0;
            while (pend != 0u) {
              uint4 v[J];
#pragma unroll
              for (int j = 0; j < J; ++j) {
                const int i = tid + j * 256, half = NB > 1 && i >= Kc ? 1 : 0, k = i - half * Kc;
                if ((pend >> j) & 1u) v[j] = ld_relaxed_gpu_v4(from + static_cast<size_t>(half * D + ks * Kc + k) * 16);
              }
#pragma unroll
              for (int j = 0; j < J; ++j) {
                const int i = tid + j * 256, half = NB > 1 && i >= Kc ? 1 : 0, k = i - half * Kc;
                if (((pend >> j) & 1u) && xg_arrived(v[j])) {
                  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + half * Cfg::HALF + k * 16), "r"(v[j].x), "r"(v[j].y), "r"(v[j].z), "r"(v[j].w) : "memory");
                  pend &= ~(1u << j);
                }
              }
              // the global timer is slow to read: look at it (and at the abort flag) only every 16th round
              if (pend != 0u && (++rounds & 15u) == 0u) {
                const uint64_t now = global_timer_ns();
                if (since == 0) since = now;
                if (*abort_flag != 0 || now - since > limit) break;
              }
            }
            // a wait that ran out in some lanes only must not leave the warp divided
            if (__any_sync(0xffffffffu, pend != 0u)) give_up(kErrWaitH, t + 1);
            if ((t & (kWideFence - 1)) == kWideFence - 1) fence_acq_rel_gpu();
            asm volatile("bar.sync 1, 256;" ::: "memory");
          }
          const long long c6 = clock();
          if (hook && prof) {
            pc[1] += c6 - c5; pc[2] += c2 - c1; pc[3] += c4 - c3; pc[4] += c3 - c2; pc[5] += c5 - c4;
          }
        }
        if (owner) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&s_out_full[slot]));
        }
        if (++slot == kRegSlots) { slot = 0; in_phase ^= 1u; }
      }
      if (hook && prof) {  // the slots of the tcgen05 kernels' phase timers that have a counterpart here
        p.err[11] = static_cast<int>(pc[4]);   // wait for the partial gates, their sum
        p.err[12] = static_cast<int>(pc[3]);   // cell, publication
        p.err[14] = static_cast<int>(pc[5]);   // outputs staged
        p.err[16] = static_cast<int>(pc[1]);   // h_t of the other CTAs, barrier
        p.err[17] = static_cast<int>(pc[2]);   // ldmatrix, mma, partial gates sent
      }
    };
    if constexpr (!EXTRA) {
      // The hooks' loop takes any call. Its second mention costs nothing, and without it these loops were scheduled worse: LSTM 16 rows D128 57.6
      // us against 55.5 (B288 T48 N2), D32 19.3 against 17.7.
      if (hooks || hist_states != CT::S || out_bf16 || clip_on) run(std::integral_constant<int, kRegHooks>{});
      else if (has_hbf && (has_cache || CELL == kElman)) run(std::integral_constant<int, kRegTrain>{});
      else if (!has_hbf && !has_cache) run(std::integral_constant<int, kRegPlain>{});
      else run(std::integral_constant<int, kRegHooks>{});
    } else {
      const bool whole = hist_states == CT::S && !out_bf16;
      if (hooks) run(std::integral_constant<int, kRegHooks>{});
      else if (whole && has_hbf && (has_cache || CELL == kElman)) run(std::integral_constant<int, kRegClipped>{});
      else if (clip_on || has_cache || has_hbf) run(std::integral_constant<int, kRegAny>{});
      else if (hist_states == 0) run(std::integral_constant<int, kRegLast>{});
      else if (out_bf16) run(std::integral_constant<int, kRegNarrow>{});
      else run(std::integral_constant<int, kRegHidden>{});
    }
    if (act) {
#pragma unroll
      for (int k = 0; k < CT::S; ++k) p.carry[static_cast<size_t>(k) * B * ND + item] = st[k];
      if (p.output_mode == 2) {
        if (out_bf16) reinterpret_cast<__nv_bfloat16*>(p.history)[item] = __float2bfloat16_rn(st[0]);
        else p.history[item] = st[0];
      }
    }
  }
  if (*abort_flag != 0) {
    // give copies that are still in flight time to land before shared memory is released
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  __syncthreads();
  cluster_sync_all();
}

template <int CELL, int KS, int NB, int KT>
int launch_fwd_wide(const FwdParams& p, const void* wx, int wx_bf16, cudaStream_t stream, bool ask) {
  using Cfg = FwdWideCfg<CELL, KS, NB, KT>;
  using CT = CellTraits<CELL>;
  constexpr int plane = Cfg::ROWS * Cfg::CHUNK;
  const int es = wx_bf16 ? 2 : 4, hes = p.out_bf16 ? 2 : 4;
  const int hist_states = p.output_mode == 0 ? CT::S : (p.output_mode == 1 ? 1 : 0);
  const bool has_cache = p.cache != nullptr && CELL != kElman;
  constexpr int steps = 4;
  const int ring = kRegSlots * (reg_round_1k(steps * CT::GW * plane * es) + reg_round_1k(steps * plane * hist_states * hes) +
                                             reg_round_1k(has_cache ? steps * plane * CT::GC * CT::CES : 0) + (p.hbf != nullptr ? reg_round_1k(steps * plane * 2) : 0));
  const int smem = Cfg::FIXED + std::max(ring, 8 * kRegScratch);
  if (smem > kRegSmemLimit) return kRegNoRoom;
  if (((reinterpret_cast<uintptr_t>(p.history) | reinterpret_cast<uintptr_t>(p.cache) | reinterpret_cast<uintptr_t>(p.hbf)) & 15u) != 0)
    return kRegNoRoom;  // bulk stores start on 16-byte boundaries
  auto kern = reg_extra<CELL>(p, hist_states, has_cache) ? frnn_fwd_wide_kernel<CELL, KS, NB, KT, true> : frnn_fwd_wide_kernel<CELL, KS, NB, KT, false>;
  const long long clusters = static_cast<long long>(p.N) * reg_batch_tiles(p.B, Cfg::ROWS) * (p.D / 32);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(clusters * KS));
  cfg.blockDim = dim3(static_cast<unsigned>(Cfg::THREADS));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];  // all CTAs wait on one another through global memory: they must be resident together
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = KS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const int rc = reg_room(reinterpret_cast<const void*>(kern), cfg, KS, clusters, 0, p.D);
  if (rc != 0 || ask) return rc != 0 ? rc : kRegTaken;
  CUtensorMap map, hist_map, cache_map, hbf_map;
  const uint64_t nd = static_cast<uint64_t>(p.N) * p.D, T = p.T, Tt = p.T_total;
  const int end = p.t0 + p.T;  // steps past the call's own are neither read nor written
  const auto tile_map = [&](CUtensorMap* m, const void* base, int bytes, int planes, int steps_end, uint64_t bs, uint64_t ps, uint64_t ss) {
    return reg_tile_map(m, base, bytes, p.D, p.N, p.B, planes, steps_end, bs, ps, ss, planes, Cfg::CHUNK, Cfg::ROWS, steps);
  };
  if (tile_map(&map, wx, es, CT::GW, end, Tt * CT::GW * nd, nd, CT::GW * nd) != 0) return -4;
  hist_map = cache_map = hbf_map = map;  // valid maps where a stream is not written
  if (hist_states > 0 && tile_map(&hist_map, p.history, hes, hist_states, end, Tt * nd, p.B * Tt * nd, nd) != 0) return -4;
  if (has_cache && tile_map(&cache_map, p.cache, CT::CES, CT::GC, p.T, T * CT::GC * nd, nd, CT::GC * nd) != 0) return -4;
  if (p.hbf != nullptr && tile_map(&hbf_map, p.hbf + nd, 2, 1, p.T, (T + 1) * nd, nd, nd) != 0) return -4;
  const int slots = wide_slots(p.T);
  const cudaError_t me = cudaMemsetAsync(p.xg_data, 0xff, static_cast<size_t>(clusters / (p.D / 32)) * slots * Cfg::ROWS * p.D * 2, stream);
  if (me != cudaSuccess) return static_cast<int>(me);
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, p, map, hist_map, cache_map, hbf_map, wx_bf16, steps, hist_states, slots));
}

template <int CELL, int KS, int NB>
int launch_fwd_wide_k(const FwdParams& p, const void* wx, int wx_bf16, cudaStream_t s, bool ask) {
  const int kt = (p.D / KS + 15) / 16;
  if constexpr (KS == 4) {  // D / 8 CTAs a group, all of them resident: 1056 units at most
    if (kt <= 12) return launch_fwd_wide<CELL, KS, NB, 12>(p, wx, wx_bf16, s, ask);
    if (kt <= 16) return launch_fwd_wide<CELL, KS, NB, 16>(p, wx, wx_bf16, s, ask);
  } else {
    if (kt <= 24) return launch_fwd_wide<CELL, KS, NB, 24>(p, wx, wx_bf16, s, ask);
    if (kt <= 28) return launch_fwd_wide<CELL, KS, NB, 28>(p, wx, wx_bf16, s, ask);
    // 128 of the 168 registers (nine warps) are fragments, some of the rest are spilled: still LSTM B16 N1 D1024 2.65 / 2.06 us per step
    if (kt <= 32) return launch_fwd_wide<CELL, KS, NB, 32>(p, wx, wx_bf16, s, ask);
  }
  return kRegNoRoom;
}

}  // namespace

// The call of a plan with `ksplit` CTAs per row tile and `rows` batch rows per group, or kRegNoRoom (its fragments do not fit the
// registers, outputs off the 16-byte grid, clusters that do not fit). Fills the exchange slots itself. `ask`: only say whether (kRegTaken).
template <int CELL>
int launch_fwd_wide_cell(const FwdParams& p, const void* wx, int wx_bf16, int rows, int ksplit, cudaStream_t s, bool ask) {
  if (ksplit == 2) return rows == 8 ? launch_fwd_wide_k<CELL, 2, 1>(p, wx, wx_bf16, s, ask) : launch_fwd_wide_k<CELL, 2, 2>(p, wx, wx_bf16, s, ask);
  if (ksplit == 4 && rows == 8) return launch_fwd_wide_k<CELL, 4, 1>(p, wx, wx_bf16, s, ask);  // where 16 rows fit so, 8 rows with ksplit 2 do
  return kRegNoRoom;
}

}  // namespace frnn
