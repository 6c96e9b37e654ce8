// Forward recurrence of narrow heads with R in the register file (see recurrent_reg.cuh).
//
// A group is one (head, 8 batch rows). Warp w of a CTA owns 8 hidden units and all of their gates: its rows of R are
// m16n8k16 A fragments, two gates of the 8 units per 16-row tile, loaded once. Per step a warp reads the operand
// round_bf16(h_{t-1}) with ldmatrix, multiplies, and each thread then holds the pre-activations of all gates of ONE unit
// for two batch rows: it runs the cell on them in registers and publishes its two values of h_t.
//   LOCAL: the CTA holds the whole head; h_t goes to the other half of a shared-memory double buffer, one mbarrier
//          arrival per warp.
//   else:  a cluster of ceil(D / 32) CTAs (an odd multiple of 16 leaves two warps of the last one without units); a quad of lanes packs the 8 batch rows of a unit into 16 bytes and sends them to
//          every CTA of the cluster with st.async on the receiver's mbarrier.
// One more warp moves data: TMA tiles of Wx in, staged outputs (history, gate cache, bf16 h) out, both under the swizzle
// that lets 8 units x 4 batch rows be read and written without bank conflicts. The compute warps' own stores of these
// outputs cost 800 cycles per step in address arithmetic and partial-line stores, their own TMA issue about as much.
//
// A group cannot overtake itself: a half of the operand double buffer is written again only after every warp has published
// the step in between, and a warp publishes after its own reads of that half.
//
// Bound: the serial chain of a step, mostly instruction issue and mma latency of one warp per scheduler: at LSTM B8 N3 D256, 1326
// cycles = operand wait 149 + Wx read and 32 mma 522 + cell 136 + publication 195 + staging of the outputs 324. The SM runs these at
// 1845 MHz (clock64 against globaltimer; the driver shows 1965), 0.71 us; the rest of the call's 0.79 us per step is the prologue
// (16 k cycles) and the launch. Per step there, against the tcgen05 kernel: 0.79 us against 1.30; GRU B16 N24 D32 0.58 against 0.68;
// Elman B16 N12 D64 0.52 against 0.66. A wait of its own for the Wx tile cost 150 cycles more (D256: 0.85 us).
#include "recurrent_reg.cuh"

namespace frnn {

namespace {

template <int CELL, int KT, bool LOCAL>
__global__ void __launch_bounds__(reg_max_threads(KT, LOCAL), reg_min_blocks(CELL, KT, LOCAL, false))
frnn_fwd_reg_kernel(const FwdParams p, const __grid_constant__ CUtensorMap wx_map, const __grid_constant__ CUtensorMap hist_map,
                    const __grid_constant__ CUtensorMap cache_map, const __grid_constant__ CUtensorMap hbf_map, const int wx_bf16,
                    const int stages_in_flight, const int hist_states) {
  const int nst = LOCAL && KT > 2 ? stages_in_flight : kRegMaxStages;  // three only in a 48-unit CTA
  using CT = CellTraits<CELL>;
  constexpr int NT = (CT::GR + 1) / 2;  // 16-row tiles: gates 2j and 2j + 1 of the warp's units
  constexpr int kHbuf = KT * 16 * 16;   // bytes of one operand buffer: [k][8 batch rows] bf16

  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t s_hbar[2];
  __shared__ int s_gave_up;  // a compute warp of this CTA has stopped waiting (the flag in global memory is an L2 round trip away)
  __shared__ __align__(8) uint64_t s_out_full[kRegMaxSlots];  // outputs of a step staged by every warp
  __shared__ __align__(8) uint64_t s_wx_full[kRegMaxStages];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane >> 2, c = lane & 3;
  const long long t_entry = clock64();
  const int D = p.D, N = p.N, T = p.T, B = p.B;
  const int nwarps = LOCAL ? (blockDim.x >> 5) - 1 : 4, U = nwarps * kRegUnitsPerWarp;
  const int C = LOCAL ? 1 : p.C;
  const int rank = LOCAL ? 0 : static_cast<int>(blockIdx.x % C), gid = blockIdx.x / C;
  const int n = gid % N, b0 = gid / N * kRegRows;
  const int unit_warps = LOCAL ? nwarps : min(nwarps, (D - rank * U) / kRegUnitsPerWarp);  // warps that own units
  uint8_t* const hbuf = smem;
  uint8_t* const wxs = smem + 2 * kHbuf;
  const int chunks = (U + kRegChunk - 1) / kRegChunk;
  const int chunk_bytes = CT::GW * kRegRows * kRegChunk * (wx_bf16 ? 2 : 4), stage_bytes = chunks * chunk_bytes;
  // Outputs of a step, staged per 32 units: history planes, gate cache, bf16 h.
  const int slots = nst + 1;
  const bool out_bf16 = p.out_bf16 != 0, has_cache = p.cache != nullptr && CELL != kElman, has_hbf = p.hbf != nullptr;
  const int hist_bytes = hist_states * (out_bf16 ? kRegPlane<2> : kRegPlane<4>);
  const int cache_bytes = has_cache ? CT::GC * kRegPlane<CT::CES> : 0;
  const int out_chunk = reg_round_1k(hist_bytes + cache_bytes + (has_hbf ? kRegPlane<2> : 0)), out_slot = chunks * out_chunk;
  uint8_t* const outs = wxs + nst * stage_bytes;
  const volatile int* abort_flag = p.err;
  const uint64_t limit = p.wait_limit_ns;
  const int mute_from = p.err[4] != 0 ? p.err[5] : 0x7fffffff;            // test hook: nobody publishes from this step on
  const uint32_t jitter = wx_bf16 ? 0u : static_cast<uint32_t>(p.err[6]); // test hook (fp32 Wx): see jitter_stall
  const bool zero_first = p.zero_first_dev != nullptr ? *p.zero_first_dev != 0 : p.slstm_zero_first != 0;
  const bool prof = p.err[3] != 0 && blockIdx.x == 0 && tid == 0;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&s_hbar[i]), (LOCAL ? nwarps : 1) + 1);  // + the I/O warp: Wx has landed
    for (int i = 0; i < slots; ++i) mbar_init(smem_u32(&s_out_full[i]), unit_warps);
    for (int s = 0; s < nst; ++s) mbar_init(smem_u32(&s_wx_full[s]), 1);
    s_gave_up = 0;
    fence_mbar_init();
    tma_prefetch_desc(&wx_map);
  }
  // operand buffer 0 = round_bf16(initial h), zero for rows past the batch and k past the head
  for (int i = tid; i < 2 * kHbuf / 4; i += blockDim.x) {
    const int k = i >> 2, b = b0 + 2 * (i & 3);
    uint32_t v = 0u;
    if (k < D) {
      const float* src = p.initial + (static_cast<size_t>(b) * N + n) * D + k;
      v = pack_bf16x2(b < B ? src[0] : 0.0f, b + 1 < B ? src[static_cast<size_t>(N) * D] : 0.0f);
    }
    reinterpret_cast<uint32_t*>(hbuf)[i] = v;
  }
  __syncthreads();
  const uint32_t h_tx = static_cast<uint32_t>(D) * kRegRows * 2u;
  if (tid == 0 && !LOCAL) {
    if (T >= 2) mbar_arrive_expect_tx(smem_u32(&s_hbar[1]), h_tx);
    if (T >= 3) mbar_arrive_expect_tx(smem_u32(&s_hbar[0]), h_tx);
  }

  if (warp == nwarps) {
    // ---------------- I/O warp: Wx tiles in, staged outputs out ----------------
    if (!LOCAL) cluster_sync_all();
    if (lane == 0) {
      auto fill = [&](int t, int s) {
        const uint32_t bar = smem_u32(&s_wx_full[s]), dst = smem_u32(wxs + s * stage_bytes);
        mbar_arrive_expect_tx(bar, stage_bytes);
        for (int i = 0; i < chunks; ++i)
          tma_load_5d(dst + i * chunk_bytes, &wx_map, bar, rank * U + i * kRegChunk, n, b0, 0, p.t0 + t);
      };
      for (int t = 0; t < nst && t < T; ++t) fill(t, t);
      int stage = 0, slot = 0, next = 1;
      uint32_t phase = 0, next_phase = 0;
      // The operand barrier of step t also stands for its Wx tile: one wait per step on the compute warps' chain, not two.
      auto announce = [&](int t) -> bool {
        if (!mbar_wait_bounded<false, true>(smem_u32(&s_wx_full[next]), next_phase & 1, limit, abort_flag)) {
          reg_report(p.err, kErrWaitWx, t);
          return false;
        }
        if (++next == nst) { next = 0; next_phase ^= 1u; }
        mbar_arrive(smem_u32(&s_hbar[t & 1]));
        return true;
      };
      // Outputs of a step staged: released by the CTA's own warps, whose waits have the plain limit, so theirs run out first. The
      // test hook makes this warp late on top of a wait that takes long anyway (the compute warps' stalls see to such waits): on
      // the direct path it costs every step of a run without it up to 80 cycles (Elman B16 N12 D64 backward 0.49 us a step -> 0.57).
      auto staged = [&](int step) -> bool {
        const uint32_t bar = smem_u32(&s_out_full[slot]);
        for (int fast = 0; fast < 64; ++fast)
          if (mbar_try_wait_spin(bar, phase)) return true;
        if (jitter != 0u) jitter_stall(jitter, 32u, static_cast<uint32_t>(step));
        return mbar_wait_bounded<false, true>(bar, phase, 2 * limit, abort_flag);
      };
      bool ok = true;
      for (int t = 1; t <= 2 && t < T && ok; ++t) ok = announce(t);
      for (int t = 0; t < T && ok; ++t) {
        if (!staged(t)) {
          reg_report(p.err, kErrWaitEpi, t);
          break;
        }
        // A warp that gave up on a wait sets the flag before it stages. Then the phase that the barrier is in may never
        // complete (another arrival would overrun its count), and a copy could be on its way into the stage: stop here.
        if (*reinterpret_cast<volatile int*>(&s_gave_up) != 0) break;
        // step t + 2 uses the barrier of step t, which every warp has left
        if (t >= 1 && t + 2 < T) ok = announce(t + 2);
        for (int i = 0; i < chunks; ++i) {
          const uint32_t src = smem_u32(outs + slot * out_slot + i * out_chunk);
          const int x = rank * U + i * kRegChunk;
          if (hist_states > 0) tma_store_5d(&hist_map, src, x, n, b0, 0, p.t0 + t);
          if (has_cache) tma_store_5d(&cache_map, src + hist_bytes, x, n, b0, 0, t);
          if (has_hbf) tma_store_5d(&hbf_map, src + hist_bytes + cache_bytes, x, n, b0, 0, t);
        }
        tma_store_commit();
        tma_store_wait_read<1>();  // the copies of step t - 1 have read their slot: see kRegMaxSlots
        if (t + nst < T) fill(t + nst, stage);
        if (++stage == nst) stage = 0;
        if (++slot == slots) { slot = 0; phase ^= 1u; }
      }
      tma_store_wait<0>();
    }
    __syncwarp();
  } else if (warp >= unit_warps) {
    cluster_sync_all();
  } else {
    const int ul = warp * kRegUnitsPerWarp + q;  // this thread's unit inside the CTA's slice
    const int d = rank * U + ul;                 // ... and inside the head
    uint32_t a[NT][KT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int kt = 0; kt < KT; ++kt)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int g = 2 * j + (r & 1), k = kt * 16 + 8 * (r >> 1) + 2 * c;
          a[j][kt][r] = (g < CT::GR && k < D)
              ? __ldg(reinterpret_cast<const uint32_t*>(p.R + ((static_cast<size_t>(g) * N + n) * D + d) * D + k)) : 0u;
        }

    const size_t ND = static_cast<size_t>(N) * D;
    bool act[2];
    float st[CT::S][2], bias[CT::GB];
#pragma unroll
    for (int g = 0; g < CT::GB; ++g) bias[g] = p.bias[(static_cast<size_t>(g) * N + n) * D + d];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int b = b0 + 2 * c + e;
      act[e] = b < B;
#pragma unroll
      for (int s = 0; s < CT::S; ++s)
        st[s][e] = act[e] ? p.initial[(static_cast<size_t>(s) * B + b) * ND + static_cast<size_t>(n) * D + d] : 0.0f;
      if (act[e] && has_hbf)
        p.hbf[(static_cast<size_t>(b) * (T + 1)) * ND + static_cast<size_t>(n) * D + d] = __float2bfloat16_rn(st[0][e]);
    }
    const bool clip_on = p.fwd_clip < INFINITY;
    const float clip = p.fwd_clip;
    const int uc = (warp & 3) * kRegUnitsPerWarp + q;  // unit inside the staged 32
    const uint32_t off_q = reg_tile_offset<2>(q, (warp & 3) * kRegUnitsPerWarp + 2 * c);
    uint8_t* const my_chunk = wxs + (warp >> 2) * chunk_bytes;
    uint8_t* const my_out = outs + (warp >> 2) * out_chunk;
    uint8_t* out = my_out;
    int slot = 0, in_stage = 0;
    bool dead = false;  // warp-uniform: after a failed wait the warp walks on without waiting
    auto give_up = [&](int code, int t) {
      if (lane == 0) reg_report(p.err, code, t);
      dead = true;
      *reinterpret_cast<volatile int*>(&s_gave_up) = 1;
    };
    float wx[CT::GW][2];
    auto read_wx = [&]() {
      const uint8_t* ws = my_chunk + in_stage * stage_bytes;
#pragma unroll
      for (int g = 0; g < CT::GW; ++g)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (wx_bf16) wx[g][e] = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(ws + g * kRegPlane<2> + reg_tile_offset<2>(2 * c + e, uc)));
          else wx[g][e] = *reinterpret_cast<const float*>(ws + g * kRegPlane<4> + reg_tile_offset<4>(2 * c + e, uc));
        }
      if (++in_stage == nst) in_stage = 0;
    };

    uint32_t peer_delta[2] = {0u, 0u};  // C <= 8: a lane of a quad sends to the peers c and c + 4
    if (!LOCAL) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (4 * i + c < C) peer_delta[i] = map_to_cta(smem_u32(smem), 4 * i + c) - smem_u32(smem);
      cluster_sync_all();
    }
    if (prof) p.err[20] = static_cast<int>(clock64() - t_entry);

    if (!mbar_wait_warp<false>(smem_u32(&s_wx_full[0]), 0, limit, abort_flag)) give_up(kErrWaitWx, 0);
    long long pc[6] = {0, 0, 0, 0, 0, 0};
    for (int t = 0; t < T; ++t) {
      if (jitter != 0u) { jitter_stall(jitter, static_cast<uint32_t>(warp), static_cast<uint32_t>(t)); __syncwarp(); }
      const int pb = t & 1;
      const long long c1 = prof ? clock64() : 0;
      if (t >= 1 && !dead && !mbar_wait_warp<!LOCAL>(smem_u32(&s_hbar[pb]), ((t - 1) >> 1) & 1, limit, abort_flag)) give_up(kErrWaitH, t);
      const long long c2 = prof ? clock64() : 0;
      read_wx();
      // One chain over k per tile, in the order of the tcgen05 kernels: the sums, and with them every output, are the same bits.
      float acc[NT][4];
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[j][r] = 0.0f;
      const uint32_t hb = smem_u32(hbuf) + pb * kHbuf + lane * 16;
#pragma unroll
      for (int k2 = 0; k2 < KT / 2; ++k2) {
        uint32_t bf[4];
        ldsm_x4_trans(hb + k2 * 512, bf);
#pragma unroll
        for (int j = 0; j < NT; ++j) mma_bf16_16816(acc[j], a[j][2 * k2], bf[0], bf[1]);
#pragma unroll
        for (int j = 0; j < NT; ++j) mma_bf16_16816(acc[j], a[j][2 * k2 + 1], bf[2], bf[3]);
      }
      const long long c3 = prof ? clock64() : 0;
      float cv[CT::GC][2];
      const bool take_i = CELL == kSLSTM && p.t0 + t == 0 && zero_first;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float ryj[CT::GR], wxj[CT::GW], sj[CT::S], cj[CT::GC];
#pragma unroll
        for (int g = 0; g < CT::GR; ++g) ryj[g] = acc[g / 2][2 * (g & 1) + e];
#pragma unroll
        for (int g = 0; g < CT::GW; ++g) wxj[g] = wx[g][e];
#pragma unroll
        for (int k = 0; k < CT::S; ++k) sj[k] = st[k][e];
        cell_forward<CELL>(ryj, wxj, bias, sj, cj, take_i);
        if (clip_on) sj[0] = fminf(fmaxf(sj[0], -clip), clip);
#pragma unroll
        for (int k = 0; k < CT::S; ++k) st[k][e] = sj[k];
#pragma unroll
        for (int k = 0; k < CT::GC; ++k) cv[k][e] = cj[k];
      }
      const uint32_t hp = pack_bf16x2(st[0][0], st[0][1]);
      const long long c4 = prof ? clock64() : 0;
      const bool publish = !dead && t + 1 < T && t < mute_from;
      const uint32_t hslot = smem_u32(hbuf) + (pb ^ 1) * kHbuf + (rank * U + warp * kRegUnitsPerWarp) * 16;
      if constexpr (LOCAL) {
        if (publish) {
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(hslot + lane * 4), "r"(hp) : "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&s_hbar[pb ^ 1]));
        }
      } else {
        uint32_t pk[4];
        gather_quad(hp, lane, pk);
        if (publish) {
          const uint32_t dst = hslot + q * 16, bar = smem_u32(&s_hbar[pb ^ 1]);
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (4 * i + c < C) st_async_v4_b32(dst + peer_delta[i], pk[0], pk[1], pk[2], pk[3], bar + peer_delta[i]);
        }
        // the operand barrier of this parity, complete since the wait above, is armed for step t + 2
        if (tid == 0 && !dead && t >= 1 && t + 2 < T) mbar_arrive_expect_tx(smem_u32(&s_hbar[pb]), h_tx);
      }
      const long long c5 = prof ? clock64() : 0;
      // outputs, while the operand of the next step is on its way
#pragma unroll
      for (int k = 0; k < CT::S; ++k)
        if (k < hist_states) {
          if (out_bf16) reg_stage_16(out + k * kRegPlane<2>, off_q, pack_bf16x2(st[k][0], st[k][1]));
          else reg_stage_f32(out + k * kRegPlane<4>, c, uc, st[k][0], st[k][1]);
        }
      if (has_cache) {
#pragma unroll
        for (int k = 0; k < CT::GC; ++k) {
          if constexpr (CT::CES == 2) {
            const __half2 hv = __floats2half2_rn(cv[k][0], cv[k][1]);
            reg_stage_16(out + hist_bytes + k * kRegPlane<2>, off_q, *reinterpret_cast<const uint32_t*>(&hv));
          } else {
            reg_stage_f32(out + hist_bytes + k * kRegPlane<4>, c, uc, cv[k][0], cv[k][1]);
          }
        }
      }
      if (has_hbf) reg_stage_16(out + hist_bytes + cache_bytes, off_q, hp);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_out_full[slot]));
      out += out_slot;
      if (++slot == slots) { slot = 0; out = my_out; }
      const long long c6 = prof ? clock64() : 0;
      if (prof) {
        pc[1] += c2 - c1; pc[2] += c3 - c2; pc[3] += c4 - c3; pc[4] += c5 - c4; pc[5] += c6 - c5;
      }
    }
    if (prof) {  // the slots of the tcgen05 kernels' phase timers that have a counterpart here
      p.err[12] = static_cast<int>(pc[3]);   // accumulators -> h_t
      p.err[13] = static_cast<int>(pc[4]);   // publication
      p.err[14] = static_cast<int>(pc[5]);   // outputs staged
      p.err[16] = static_cast<int>(pc[1]);   // operand wait
      p.err[17] = static_cast<int>(pc[2]);   // Wx read, ldmatrix, mma
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (!act[e]) continue;
      const size_t item = static_cast<size_t>(b0 + 2 * c + e) * ND + static_cast<size_t>(n) * D + d;
#pragma unroll
      for (int k = 0; k < CT::S; ++k) p.carry[static_cast<size_t>(k) * B * ND + item] = st[k][e];
      if (p.output_mode == 2) {
        if (out_bf16) reinterpret_cast<__nv_bfloat16*>(p.history)[item] = __float2bfloat16_rn(st[0][e]);
        else p.history[item] = st[0][e];
      }
    }
  }
  if (*abort_flag != 0) {
    // give copies that are still in flight time to land before shared memory is released
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  __syncthreads();
  if (!LOCAL) cluster_sync_all();
}

template <int CELL, int KT, bool LOCAL>
int launch_fwd_reg(const FwdParams& p, const void* wx, int wx_bf16, cudaStream_t stream, bool ask) {
  using CT = CellTraits<CELL>;
  const int U = LOCAL ? p.D : kRegClusterUnits, es = wx_bf16 ? 2 : 4;
  const int plane = kRegRows * kRegChunk;
  const int stage = reg_chunks(U) * CT::GW * plane * es;
  const int hist_states = p.output_mode == 0 ? CT::S : (p.output_mode == 1 ? 1 : 0);
  const int hes = p.out_bf16 ? 2 : 4;
  const bool has_cache = p.cache != nullptr && CELL != kElman;
  const int out_slot = reg_chunks(U) * reg_round_1k(plane * (hist_states * hes + (has_cache ? CT::GC * CT::CES : 0) + (p.hbf != nullptr ? 2 : 0)));
  // prefetch depth: 4 steps, 3 where only that lets two CTAs share an SM
  const auto bytes = [&](int st) { return 2 * KT * 16 * 16 + st * stage + (st + 1) * out_slot; };
  const int nst = LOCAL && KT > 2 ? reg_stages(bytes(kRegMaxStages), bytes(kRegMaxStages - 1)) : kRegMaxStages;
  const int smem = bytes(nst);
  if (smem > kRegSmemLimit) return -2;
  // bulk stores start on 16-byte boundaries; the tcgen05 kernels write these outputs with plain stores
  if (((reinterpret_cast<uintptr_t>(p.history) | reinterpret_cast<uintptr_t>(p.cache) | reinterpret_cast<uintptr_t>(p.hbf)) & 15u) != 0)
    return kRegNoRoom;
  auto kern = frnn_fwd_reg_kernel<CELL, KT, LOCAL>;
  FwdParams q = p;
  q.C = (p.D + U - 1) / U;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(p.N * reg_batch_tiles(p.B) * q.C));
  cfg.blockDim = dim3(static_cast<unsigned>(U / kRegUnitsPerWarp * 32 + 32));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(q.C);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = LOCAL ? 0 : 1;
  // whether the call is taken at all comes first: one that is not pays for nothing else
  const int rc = reg_room(reinterpret_cast<const void*>(kern), cfg, q.C, p.N, p.B, p.D);
  if (rc != 0 || ask) return rc != 0 ? rc : kRegTaken;
  CUtensorMap map, hist_map, cache_map, hbf_map;
  const uint64_t nd = static_cast<uint64_t>(p.N) * p.D, T = p.T, Tt = p.T_total;
  if (reg_tile_map(&map, wx, es, p.D, p.N, p.B, CT::GW, p.T_total, Tt * CT::GW * nd, nd, CT::GW * nd, CT::GW) != 0) return -4;
  hist_map = cache_map = hbf_map = map;  // valid maps where a stream is not written
  if (hist_states > 0 &&
      reg_tile_map(&hist_map, p.history, hes, p.D, p.N, p.B, hist_states, p.T_total, Tt * nd, p.B * Tt * nd, nd, hist_states) != 0)
    return -4;
  if (has_cache && reg_tile_map(&cache_map, p.cache, CT::CES, p.D, p.N, p.B, CT::GC, p.T, T * CT::GC * nd, nd, CT::GC * nd, CT::GC) != 0)
    return -4;
  if (p.hbf != nullptr && reg_tile_map(&hbf_map, p.hbf + nd, 2, p.D, p.N, p.B, 1, p.T, (T + 1) * nd, nd, nd, 1) != 0) return -4;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, q, map, hist_map, cache_map, hbf_map, wx_bf16, nst, hist_states));
}

template <int CELL>
int launch_fwd_reg_cell(const FwdParams& p, const void* wx, int wx_bf16, cudaStream_t s, bool ask) {
  switch (reg_k_tiles(p.D)) {
    case 2: return launch_fwd_reg<CELL, 2, true>(p, wx, wx_bf16, s, ask);
    case 4:
      return reg_local(p.D) ? launch_fwd_reg<CELL, 4, true>(p, wx, wx_bf16, s, ask)
                                  : launch_fwd_reg<CELL, 4, false>(p, wx, wx_bf16, s, ask);
    case 6: return launch_fwd_reg<CELL, 6, false>(p, wx, wx_bf16, s, ask);
    case 8: return launch_fwd_reg<CELL, 8, false>(p, wx, wx_bf16, s, ask);
    case 10: return launch_fwd_reg<CELL, 10, false>(p, wx, wx_bf16, s, ask);
    case 12: return launch_fwd_reg<CELL, 12, false>(p, wx, wx_bf16, s, ask);
    case 14: return launch_fwd_reg<CELL, 14, false>(p, wx, wx_bf16, s, ask);
    case 16: return launch_fwd_reg<CELL, 16, false>(p, wx, wx_bf16, s, ask);
    default: return -2;
  }
}

}  // namespace

int forward_reg_dispatch(int cell, const FwdParams& p, const void* wx, int wx_bf16, cudaStream_t s, bool ask) {
  switch (cell) {
    case kLSTM: return launch_fwd_reg_cell<kLSTM>(p, wx, wx_bf16, s, ask);
    case kSLSTM: return launch_fwd_reg_cell<kSLSTM>(p, wx, wx_bf16, s, ask);
    case kGRU: return launch_fwd_reg_cell<kGRU>(p, wx, wx_bf16, s, ask);
    case kElman: return launch_fwd_reg_cell<kElman>(p, wx, wx_bf16, s, ask);
    default: return -1;
  }
}

}  // namespace frnn
