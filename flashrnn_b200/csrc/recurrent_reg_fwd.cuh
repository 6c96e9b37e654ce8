// Forward recurrence of narrow heads with R in the register file (see recurrent_reg.cuh).
//
// A group is one (head, 8, 16 or 24 batch rows: NB column tiles). Warp w of a CTA owns 4 hidden units (Elman: 8) and all of their
// gates: its rows of R are m16n8k16 A fragments, the four gates of 4 units per 16-row tile, loaded once. Per step a warp reads the
// operand round_bf16(h_{t-1}) with ldmatrix, multiplies, and two lanes swap halves, so that each thread holds the pre-activations of
// all gates of ONE item (unit, batch row) per column tile: it runs the cell on them in registers and publishes its value of h_t.
//   LOCAL: the CTA holds the whole head; h_t goes to the other half of a shared-memory double buffer, one CTA barrier a step.
//   else:  a cluster of ceil(D / 32) CTAs (an odd multiple of 16 leaves four warps of the last one without units); the word of two
//          batch rows of a unit goes to every CTA of the cluster with st.async on the receiver's mbarrier, half of the peers from
//          either lane of the pair. Packets of 16 bytes, put together by a quad of lanes, were 3 to 8 % slower on every cell but the
//          Elman with more than four peers (GATHER).
// One more warp moves data: TMA tiles of Wx in, staged outputs (history, gate cache, bf16 h) out, both under the swizzle
// that lets units x batch rows be read and written without bank conflicts, several steps per transfer (reg_transfer_steps). The
// compute warps' own stores of these outputs cost 800 cycles per step in address arithmetic and partial-line stores, their own
// TMA issue about as much. The loop over the steps is compiled for the outputs that the call has (kRegHooks ...):
// flags and offsets at run time were 5 to 25 % of a step, the hooks' tests alone 3 to 6 (LSTM B9 T256 N1 D512, us: hidden states alone 337
// in one loop for everything, 271 in their own; with a clip in training 348 / 298).
//
// A group cannot overtake itself: a half of the operand double buffer is written again only after every warp has published
// the step in between, and a warp publishes after its own reads of that half.
//
// Bound: the serial chain of a step: instruction issue (4.5 cycles for each instruction of a lone warp), mma latency (24 cycles a
// dependent pair, 13 to 14.5 of a scheduler each), DSMEM flight (400), one successful mbarrier wait (150 to 180). LSTM B8 N3 D256, cycles: Wx read
// and operand wait 268, ldmatrix and mma 433, cell 107, publication 242, staging 201; the prologue is 10 k.
// us per step before (8 units a warp, packets, a transfer per step) and now, kernel and prologue: LSTM B8 N3 D256 0.80 / 0.64; LSTM
// B16 N4 D128 0.71 / 0.50; sLSTM there 0.85 / 0.59; LSTM B8 N1 D64 fp32 0.64 / 0.42; GRU B16 N24 D32 0.58 / 0.30; Elman B16 N12 D64
// 0.53 / 0.34. Against the tcgen05 kernels, which had these before: LSTM B256 N4 D128 (16 rows) 1.30 / 1.03; B8 N1 D384 1.68 / 0.78,
// D512 2.07 / 1.10; B64 N3 D256 (24 rows) 1.47 / 0.97.
#pragma once

#include <algorithm>
#include <type_traits>

#include "recurrent_reg.cuh"

namespace frnn {

namespace {

// DENSE: one more CTA on the SM where all groups run at once with it only (see launch_fwd_reg).
template <int CELL, int KT, bool LOCAL, int NB, bool DENSE = false>
struct FwdRegCfg {
  static constexpr int UPW = CELL == kElman ? 8 : 4;         // units of a warp: one 16-row tile holds all gates of four
  static constexpr int IT = UPW / 4, NI = NB * IT;           // items (unit, batch row) of a thread, per column tile and in all
  static constexpr int ROWS = NB * kRegRows;
  static constexpr int U = LOCAL ? KT * 16 : 32;             // units of a CTA
  static constexpr int MAX_C = LOCAL ? 1 : KT / 2;
  static constexpr int THREADS = (U / UPW + 1) * 32;
  // h_t goes to a peer as the words of two batch rows, or (GATHER) as packets of eight that a quad of lanes puts together
  static constexpr bool GATHER = UPW == 8 && MAX_C > 4;
  // CTAs per SM the register budget is cut for. Elman: four compute warps; 124 registers instead of 132 at 256 units let a third CTA in (B304
  // T64 D224 59 / 47 us, where two take 16 rows a group), and cost nothing where it has no work.
  static constexpr int MIN_BLOCKS = LOCAL ? (KT <= 2 ? 4 : (CELL == kSLSTM ? 1 : 2))
                                          : ((CELL == kElman && KT <= 16 && NB == 1) || (DENSE && KT == 4) ? 3 : (KT <= 8 || CELL == kElman || DENSE ? 2 : 1));
};

template <int CELL, int KT, bool LOCAL, int NB, bool DENSE, bool EXTRA>
__global__ void __launch_bounds__(FwdRegCfg<CELL, KT, LOCAL, NB, DENSE>::THREADS, FwdRegCfg<CELL, KT, LOCAL, NB, DENSE>::MIN_BLOCKS)
frnn_fwd_reg_kernel(const FwdParams p, const __grid_constant__ CUtensorMap wx_map, const __grid_constant__ CUtensorMap hist_map,
                    const __grid_constant__ CUtensorMap cache_map, const __grid_constant__ CUtensorMap hbf_map, const int wx_bf16,
                    const int ring_steps, const int hist_states) {
  using Cfg = FwdRegCfg<CELL, KT, LOCAL, NB, DENSE>;
  using CT = CellTraits<CELL>;
  constexpr int UPW = Cfg::UPW, IT = Cfg::IT, NI = Cfg::NI, CHUNK = kRegChunk, ROWS = Cfg::ROWS, U = Cfg::U, nwarps = U / UPW;
  constexpr int kPlane2 = ROWS * CHUNK * 2, kPlane4 = ROWS * CHUNK * 4, kPlaneC = ROWS * CHUNK * CT::CES;
  constexpr int kHalf = KT * 16 * 16;    // bytes of one column tile of the operand: [k][8 batch rows] bf16
  constexpr int kHbuf = NB * kHalf;      // ... of one operand buffer
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t s_hbar[2];
  __shared__ int s_gave_up;  // a compute warp of this CTA has stopped waiting (the flag in global memory is an L2 round trip away)
  __shared__ __align__(8) uint64_t s_out_full[kRegSlots];  // outputs of a transfer staged by every warp
  __shared__ __align__(8) uint64_t s_wx_full[kRegSlots];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane >> 2, c = lane & 3, hi = lane >> 4;
  const long long t_entry = clock64();
  const int D = p.D, N = p.N, T = p.T, B = p.B;
  const int C = LOCAL ? 1 : p.C;
  const int rank = LOCAL ? 0 : static_cast<int>(blockIdx.x % C), gid = blockIdx.x / C;
  const int n = gid % N, b0 = gid / N * ROWS;
  const int unit_warps = LOCAL ? nwarps : min(nwarps, (D - rank * U) / UPW);  // warps that own units
  uint8_t* const hbuf = smem;
  uint8_t* const wxs = smem + reg_round_1k(2 * kHbuf);
  constexpr int chunks = (U + CHUNK - 1) / CHUNK;
  const int chunk_bytes = CT::GW * (wx_bf16 ? kPlane2 : kPlane4), stage_bytes = chunks * ring_steps * chunk_bytes;
  // A transfer of inputs: [chunk of units][step][gate]; of outputs: per chunk of units the history planes of its steps, the gate
  // cache of its steps, bf16 h of its steps.
  const bool out_bf16 = p.out_bf16 != 0, has_cache = p.cache != nullptr && CELL != kElman, has_hbf = p.hbf != nullptr;
  const int hist_bytes = hist_states * (out_bf16 ? kPlane2 : kPlane4);
  const int cache_bytes = has_cache ? CT::GC * kPlaneC : 0;
  const int out_chunk = reg_round_1k(ring_steps * (hist_bytes + cache_bytes + (has_hbf ? kPlane2 : 0))), out_slot = chunks * out_chunk;
  uint8_t* const outs = wxs + reg_round_1k(kRegSlots * stage_bytes);
  const volatile int* abort_flag = p.err;
  const uint64_t limit = p.wait_limit_ns;
  const bool zero_first = p.zero_first_dev != nullptr ? *p.zero_first_dev != 0 : p.slstm_zero_first != 0;
  // hooks of the caller: phase timers; nobody publishes from a step on; delays (fp32 Wx: see jitter_stall)
  const bool prof = p.err[3] != 0 && blockIdx.x == 0 && tid == 0;
  const int mute_from = p.err[4] != 0 ? p.err[5] : 0x7fffffff;
  const uint32_t jitter = wx_bf16 ? 0u : static_cast<uint32_t>(p.err[6]);
  const bool hooks = p.err[3] != 0 || p.err[4] != 0 || (jitter != 0u && p.err[7] == 0);  // err[7]: only the I/O warp is late

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&s_hbar[i]), 1);
    for (int i = 0; i < kRegSlots; ++i) {
      mbar_init(smem_u32(&s_out_full[i]), unit_warps);
      mbar_init(smem_u32(&s_wx_full[i]), 1);
    }
    s_gave_up = 0;
    fence_mbar_init();
    tma_prefetch_desc(&wx_map);
  }
  // operand buffer 0 = round_bf16(initial h), zero for rows past the batch and k past the head; buffer 1 zero
  reg_fill_operand<NB, KT>(hbuf, p.initial + static_cast<size_t>(n) * D, static_cast<size_t>(N) * D, b0, B, D, tid, blockDim.x);
  __syncthreads();
  const uint32_t h_tx = static_cast<uint32_t>(D) * ROWS * 2u;
  if (tid == 0 && !LOCAL) {
    if (T >= 2) mbar_arrive_expect_tx(smem_u32(&s_hbar[1]), h_tx);
    if (T >= 3) mbar_arrive_expect_tx(smem_u32(&s_hbar[0]), h_tx);
  }

  if (warp == nwarps) {
    // ---------------- I/O warp: Wx tiles in, staged outputs out ----------------
    if (!LOCAL) cluster_sync_all();
    if (lane == 0) {
      auto fill = [&](int t, int s) {  // the inputs of the steps t .. t + ring_steps - 1
        const uint32_t bar = smem_u32(&s_wx_full[s]), dst = smem_u32(wxs + s * stage_bytes);
        mbar_arrive_expect_tx(bar, stage_bytes);
#pragma unroll
        for (int i = 0; i < chunks; ++i)
          tma_load_5d(dst + i * ring_steps * chunk_bytes, &wx_map, bar, rank * U + i * CHUNK, n, b0, 0, p.t0 + t);
      };
      for (int i = 0; i < kRegSlots && i * ring_steps < T; ++i) fill(i * ring_steps, i);
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
      for (int t = 0; t < T; t += ring_steps) {
        if (!staged(t)) {
          reg_report(p.err, kErrWaitEpi, t);
          break;
        }
        // A warp that gave up on a wait sets the flag before it stages. Then the phase that the barrier is in may never
        // complete (another arrival would overrun its count), and a copy could be on its way into the stage: stop here.
        if (*reinterpret_cast<volatile int*>(&s_gave_up) != 0) break;
#pragma unroll
        for (int i = 0; i < chunks; ++i) {
          const uint32_t src = smem_u32(outs + slot * out_slot + i * out_chunk);
          const int x = rank * U + i * CHUNK;
          if (hist_states > 0) tma_store_5d(&hist_map, src, x, n, b0, 0, p.t0 + t);
          if (has_cache) tma_store_5d(&cache_map, src + ring_steps * hist_bytes, x, n, b0, 0, t);
          if (has_hbf) tma_store_5d(&hbf_map, src + ring_steps * (hist_bytes + cache_bytes), x, n, b0, 0, t);
        }
        tma_store_commit();
        // A warp that stages into this slot again has read the inputs asked for below, after these copies have read the slot.
        tma_store_wait_read<0>();
        if (t + kRegSlots * ring_steps < T) fill(t + kRegSlots * ring_steps, slot);
        if (++slot == kRegSlots) { slot = 0; phase ^= 1u; }
      }
      tma_store_wait<0>();
    }
    __syncwarp();
  } else if (warp >= unit_warps) {
    cluster_sync_all();
  } else {
    // The items of a thread are one unit of one batch row of each column tile: lanes 0 - 15 have the even rows, 16 - 31 the
    // odd ones. Elman: one unit of two neighbouring rows, the rows 8 - 15 of its fragments are zero.
    const int uq = UPW == 4 ? q & 3 : q;
    const int ul = warp * UPW + uq;  // this thread's unit inside the CTA's slice
    const int d = rank * U + ul;     // ... and inside the head
    auto item_row = [&](int i) { return i / IT * 8 + 2 * c + (UPW == 4 ? hi : i % IT); };
    uint32_t a[KT][4];
    // The I/O warp of a cluster asks for the first tiles after the cluster has met: the ring is scratch until then.
    reg_load_rows<KT, UPW, CT::GR>(p.R + (static_cast<size_t>(n) * D + rank * U + warp * UPW) * D, static_cast<size_t>(N) * D * D, D, D,
                                   smem_u32(wxs) + warp * kRegScratch, lane, !LOCAL && (reinterpret_cast<uintptr_t>(p.R) & 15u) == 0, a);

    const size_t ND = static_cast<size_t>(N) * D;
    bool act[NI];
    float st[CT::S][NI], bias[CT::GB];
#pragma unroll
    for (int g = 0; g < CT::GB; ++g) bias[g] = p.bias[(static_cast<size_t>(g) * N + n) * D + d];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int b = b0 + item_row(i);
      act[i] = b < B;
#pragma unroll
      for (int s = 0; s < CT::S; ++s)
        st[s][i] = act[i] ? p.initial[(static_cast<size_t>(s) * B + b) * ND + static_cast<size_t>(n) * D + d] : 0.0f;
      if (act[i] && has_hbf)
        p.hbf[(static_cast<size_t>(b) * (T + 1)) * ND + static_cast<size_t>(n) * D + d] = __float2bfloat16_rn(st[0][i]);
    }
    const bool clip_on = p.fwd_clip < INFINITY;
    const float clip = p.fwd_clip;
    const int uc = ul % CHUNK;  // unit inside the staged chunk
    // offsets of the thread's items in a plane; those of the second column tile are 8 rows further
    uint32_t off2[IT], off4[IT];
#pragma unroll
    for (int i = 0; i < IT; ++i) {
      off2[i] = reg_tile_offset<2, CHUNK>(item_row(i), uc);
      off4[i] = reg_tile_offset<4, CHUNK>(item_row(i), uc);
    }
    const uint32_t my_chunk = smem_u32(wxs) + ul / CHUNK * ring_steps * chunk_bytes, my_out = smem_u32(outs) + ul / CHUNK * out_chunk;
    bool dead = false;  // warp-uniform: after a failed wait the warp walks on without waiting
    auto give_up = [&](int code, int t) {
      if (lane == 0) reg_report(p.err, code, t);
      dead = true;
      *reinterpret_cast<volatile int*>(&s_gave_up) = 1;
    };

    // Peers of a lane. Words: lanes 16 apart hold the two rows of a word between them; of two column tiles each packs one and sends it
    // to every peer, of a single one both pack the same word and share the peers. Packets: the quad shares the peers.
    constexpr int SENDERS = Cfg::GATHER ? 4 : 1, NS = (Cfg::MAX_C + SENDERS - 1) / SENDERS;
    const int sender = Cfg::GATHER ? c : 0;
    uint32_t peer_delta[NS];
    if (!LOCAL) {
#pragma unroll
      for (int i = 0; i < NS; ++i)
        peer_delta[i] = SENDERS * i + sender < C ? map_to_cta(smem_u32(smem), SENDERS * i + sender) - smem_u32(smem) : 0u;
      cluster_sync_all();
    }
    if (prof) p.err[20] = static_cast<int>(clock64() - t_entry);

    // The steps, compiled for what the call writes, and for anything (with the hooks): see above.
    auto run = [&](auto mode_tag) {
      constexpr int MODE = decltype(mode_tag)::value;
      constexpr bool hook = MODE == kRegHooks, any = hook || MODE == kRegAny, train = MODE == kRegTrain || MODE == kRegClipped;
      const bool save = any ? has_cache : train && CELL != kElman, keep_h = any ? has_hbf : train;
      const bool narrow = any ? out_bf16 : MODE == kRegNarrow, clipped = any ? clip_on : MODE == kRegClipped;
      const int states = any || MODE == kRegNarrow ? hist_states : (MODE == kRegHidden ? 1 : (MODE == kRegLast ? 0 : CT::S));
      const int hist_step = any || MODE == kRegNarrow ? hist_bytes : states * kPlane4, cache_step = any ? cache_bytes : (save ? CT::GC * kPlaneC : 0);
      long long pc[6] = {0, 0, 0, 0, 0, 0};
      auto clock = [&]() -> long long { return hook && prof ? clock64() : 0; };
      uint32_t hb = smem_u32(hbuf), hb_next = hb + kHbuf;  // operand of this step, of the next
      int slot = 0;
      uint32_t in_phase = 0;
      for (int t0 = 0; t0 < T; t0 += ring_steps) {
        if (!dead && !mbar_wait_warp<false>(smem_u32(&s_wx_full[slot]), in_phase, limit, abort_flag)) give_up(kErrWaitWx, t0);
        const int t_end = min(T, t0 + ring_steps);
        uint32_t in = my_chunk + slot * stage_bytes, out_h = my_out + slot * out_slot;
        uint32_t out_c = out_h + ring_steps * hist_step, out_b = out_c + ring_steps * cache_step;
        for (int t = t0; t < t_end; ++t) {
          if (hook && jitter != 0u) { jitter_stall(jitter, static_cast<uint32_t>(warp), static_cast<uint32_t>(t)); __syncwarp(); }
          const long long c1 = clock();
          float wx[CT::GW][NI];
          if (wx_bf16) {
#pragma unroll
            for (int g = 0; g < CT::GW; ++g)
#pragma unroll
              for (int i = 0; i < NI; ++i) wx[g][i] = __uint_as_float(lds_u16(in + off2[i % IT] + g * kPlane2 + i / IT * (8 * CHUNK * 2)) << 16);
          } else {
#pragma unroll
            for (int g = 0; g < CT::GW; ++g)
#pragma unroll
              for (int i = 0; i < NI; ++i) wx[g][i] = lds_f32(in + off4[i % IT] + g * kPlane4 + i / IT * (8 * CHUNK * 4));
          }
          in += wx_bf16 ? CT::GW * kPlane2 : CT::GW * kPlane4;
          if constexpr (LOCAL) {
            // h of every warp; what a silenced step leaves out is waited for on a barrier that nobody arrives at
            if (t >= 1) asm volatile("bar.sync 1, %0;" ::"n"(nwarps * 32) : "memory");
            if (hook && t > mute_from && !dead && !mbar_wait_warp<false>(smem_u32(&s_hbar[0]), 0, limit, abort_flag)) give_up(kErrWaitH, t);
          } else {
            if (t >= 1 && !dead && !mbar_wait_warp<true>(smem_u32(&s_hbar[t & 1]), ((t - 1) >> 1) & 1, limit, abort_flag)) give_up(kErrWaitH, t);
          }
          const long long c2 = clock();
          // One chain over k per tile, in the order of the tcgen05 kernels: the sums, and with them every output, are the same bits.
          float acc[NB][4];
#pragma unroll
          for (int j = 0; j < NB; ++j)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[j][r] = 0.0f;
#pragma unroll
          for (int k2 = 0; k2 < KT / 2; ++k2) {
            uint32_t bf[NB][4];
#pragma unroll
            for (int j = 0; j < NB; ++j) ldsm_x4_trans(hb + lane * 16 + j * kHalf + k2 * 512, bf[j]);
#pragma unroll
            for (int j = 0; j < NB; ++j) mma_bf16_16816(acc[j], a[2 * k2], bf[j][0], bf[j][1]);
#pragma unroll
            for (int j = 0; j < NB; ++j) mma_bf16_16816(acc[j], a[2 * k2 + 1], bf[j][2], bf[j][3]);
          }
          if constexpr (KT % 2 == 1) {
#pragma unroll
            for (int j = 0; j < NB; ++j) {
              uint32_t b0w, b1w;
              ldsm_x2_trans(hb + j * kHalf + (KT - 1) * 256 + (lane & 15) * 16, b0w, b1w);
              mma_bf16_16816(acc[j], a[KT - 1], b0w, b1w);
            }
          }
          // All gates of an item to one thread: rows q and q + 8 of a fragment are the gates hi and 2 + hi of unit q & 3, the lanes 16
          // apart swap the column the other one keeps.
          float ry[4][NI];
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            if constexpr (UPW == 4) {
              const float x0 = __shfl_xor_sync(0xffffffffu, hi ? acc[j][0] : acc[j][1], 16);
              const float x1 = __shfl_xor_sync(0xffffffffu, hi ? acc[j][2] : acc[j][3], 16);
              ry[0][j] = hi ? x0 : acc[j][0];
              ry[1][j] = hi ? acc[j][1] : x0;
              ry[2][j] = hi ? x1 : acc[j][2];
              ry[3][j] = hi ? acc[j][3] : x1;
            } else {
              ry[0][2 * j] = acc[j][0];
              ry[0][2 * j + 1] = acc[j][1];
            }
          }
          const long long c3 = clock();
          float cv[CT::GC][NI];
          const bool take_i = CELL == kSLSTM && p.t0 + t == 0 && zero_first;
#pragma unroll
          for (int i = 0; i < NI; ++i) {
            float ryj[CT::GR], wxj[CT::GW], sj[CT::S], cj[CT::GC];
#pragma unroll
            for (int g = 0; g < CT::GR; ++g) ryj[g] = ry[g][i];
#pragma unroll
            for (int g = 0; g < CT::GW; ++g) wxj[g] = wx[g][i];
#pragma unroll
            for (int k = 0; k < CT::S; ++k) sj[k] = st[k][i];
            cell_forward<CELL>(ryj, wxj, bias, sj, cj, take_i);
            if (clipped) sj[0] = fminf(fmaxf(sj[0], -clip), clip);
#pragma unroll
            for (int k = 0; k < CT::S; ++k) st[k][i] = sj[k];
#pragma unroll
            for (int k = 0; k < CT::GC; ++k) cv[k][i] = cj[k];
          }
          const long long c4 = clock();
          const bool publish = t + 1 < T && !(hook && (dead || t >= mute_from));
          const uint32_t hslot = hb_next + (rank * U + warp * UPW + uq) * 16;
          if constexpr (LOCAL) {
            if (publish) {
#pragma unroll
              for (int i = 0; i < NI; ++i) sts_u16(hslot + i / IT * kHalf + (item_row(i) & 7) * 2, bf16_bits(st[0][i]));
            }
          } else {
            const uint32_t bar = smem_u32(&s_hbar[(t + 1) & 1]);
            if constexpr (UPW == 8) {
#pragma unroll
              for (int j = 0; j < NB; ++j) {
                const uint32_t w = pack_bf16x2(st[0][2 * j], st[0][2 * j + 1]), dst = hslot + j * kHalf;
                uint32_t pk[4];
                if constexpr (Cfg::GATHER) gather_quad(w, lane, pk);
                if (publish && !dead) {
#pragma unroll
                  for (int i = 0; i < NS; ++i) {
                    if (SENDERS * i + sender >= C) continue;
                    if constexpr (Cfg::GATHER) st_async_v4_b32(dst + peer_delta[i], pk[0], pk[1], pk[2], pk[3], bar + peer_delta[i]);
                    else st_async_b32(dst + c * 4 + peer_delta[i], w, bar + peer_delta[i]);
                  }
                }
              }
            } else {
#pragma unroll
              for (int j = 0; j < NB; j += 2) {
                const bool two = j + 1 < NB;
                const float mine = two && hi ? st[0][two ? j + 1 : j] : st[0][j];
                const float other = __shfl_xor_sync(0xffffffffu, two && !hi ? st[0][two ? j + 1 : j] : st[0][j], 16);
                const uint32_t w = pack_bf16x2(hi ? other : mine, hi ? mine : other);
                if (publish && !dead) {
                  if (two) {
                    const uint32_t dst = hslot + (j + hi) * kHalf + c * 4;
#pragma unroll
                    for (int i = 0; i < NS; ++i)
                      if (i < C) st_async_b32(dst + peer_delta[i], w, bar + peer_delta[i]);
                  } else {
                    const uint32_t dst = hslot + j * kHalf + c * 4;
#pragma unroll
                    for (int i = 0; i < NS; i += 2) {
                      const uint32_t delta = hi ? peer_delta[i + 1 < NS ? i + 1 : i] : peer_delta[i];
                      if (i + hi < C) st_async_b32(dst + delta, w, bar + delta);
                    }
                  }
                }
              }
            }
          }
          const long long c5 = clock();
          // outputs, while the operand of the next step is on its way
#pragma unroll
          for (int i = 0; i < NI; ++i) {
            const int e = i % IT, far2 = i / IT * (8 * CHUNK * 2), far4 = i / IT * (8 * CHUNK * 4);
#pragma unroll
            for (int k = 0; k < CT::S; ++k)
              if (k < states) {
                if (narrow) sts_u16(out_h + off2[e] + k * kPlane2 + far2, bf16_bits(st[k][i]));
                else sts_f32(out_h + off4[e] + k * kPlane4 + far4, st[k][i]);
              }
            if (save) {
#pragma unroll
              for (int k = 0; k < CT::GC; ++k) {
                if constexpr (CT::CES == 2) sts_u16(out_c + off2[e] + k * kPlane2 + far2, __half_as_ushort(__float2half_rn(cv[k][i])));
                else sts_f32(out_c + off4[e] + k * kPlane4 + far4, cv[k][i]);
              }
            }
            if (keep_h) sts_u16(out_b + off2[e] + far2, bf16_bits(st[0][i]));
          }
          out_h += hist_step;
          out_c += cache_step;
          out_b += kPlane2;
          // the operand barrier of this parity, complete since the wait above, is armed for step t + 2
          if (!LOCAL && tid == 0 && !dead && t >= 1 && t + 2 < T) mbar_arrive_expect_tx(smem_u32(&s_hbar[t & 1]), h_tx);
          const uint32_t swap = hb;
          hb = hb_next;
          hb_next = swap;
          const long long c6 = clock();
          if (hook && prof) {
            pc[1] += c2 - c1; pc[2] += c3 - c2; pc[3] += c4 - c3; pc[4] += c5 - c4; pc[5] += c6 - c5;
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&s_out_full[slot]));
        if (++slot == kRegSlots) { slot = 0; in_phase ^= 1u; }
      }
      if (hook && prof) {  // the slots of the tcgen05 kernels' phase timers that have a counterpart here
        p.err[12] = static_cast<int>(pc[3]);   // accumulators -> h_t
        p.err[13] = static_cast<int>(pc[4]);   // publication
        p.err[14] = static_cast<int>(pc[5]);   // outputs staged
        p.err[16] = static_cast<int>(pc[1]);   // Wx read, operand wait
        p.err[17] = static_cast<int>(pc[2]);   // ldmatrix, mma
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
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      if (!act[i]) continue;
      const size_t item = static_cast<size_t>(b0 + item_row(i)) * ND + static_cast<size_t>(n) * D + d;
#pragma unroll
      for (int k = 0; k < CT::S; ++k) p.carry[static_cast<size_t>(k) * B * ND + item] = st[k][i];
      if (p.output_mode == 2) {
        if (out_bf16) reinterpret_cast<__nv_bfloat16*>(p.history)[item] = __float2bfloat16_rn(st[0][i]);
        else p.history[item] = st[0][i];
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

// Runs the call, or (ask) only says whether it would: kRegTaken / kRegNoRoom.
template <int CELL, int KT, bool LOCAL, int NB, bool DENSE = false>
int launch_fwd_reg(const FwdParams& p, const void* wx, int wx_bf16, cudaStream_t stream, bool ask, long long rival_groups = 0) {
  using Cfg = FwdRegCfg<CELL, KT, LOCAL, NB, DENSE>;
  using CT = CellTraits<CELL>;
  constexpr int U = Cfg::U, ROWS = Cfg::ROWS, CHUNK = kRegChunk, plane = ROWS * CHUNK, chunks = (U + CHUNK - 1) / CHUNK;
  const int es = wx_bf16 ? 2 : 4;
  const int stage = chunks * CT::GW * plane * es;
  const int hist_states = p.output_mode == 0 ? CT::S : (p.output_mode == 1 ? 1 : 0);
  const int hes = p.out_bf16 ? 2 : 4;
  const bool has_cache = p.cache != nullptr && CELL != kElman;
  const int out_step = plane * (hist_states * hes + (has_cache ? CT::GC * CT::CES : 0) + (p.hbf != nullptr ? 2 : 0));
  constexpr int fixed = reg_round_1k(2 * NB * KT * 16 * 16);
  const int steps = reg_transfer_steps(fixed, stage + chunks * out_step, Cfg::MIN_BLOCKS);
  const int ring = reg_round_1k(kRegSlots * steps * stage) + kRegSlots * chunks * reg_round_1k(steps * out_step);
  const int smem = fixed + std::max(ring, LOCAL ? 0 : (Cfg::THREADS / 32 - 1) * kRegScratch);
  if (smem > kRegSmemLimit) return kRegNoRoom;
  // bulk stores start on 16-byte boundaries; the tcgen05 kernels write these outputs with plain stores
  if (((reinterpret_cast<uintptr_t>(p.history) | reinterpret_cast<uintptr_t>(p.cache) | reinterpret_cast<uintptr_t>(p.hbf)) & 15u) != 0)
    return kRegNoRoom;
  const bool extra = reg_extra<CELL>(p, hist_states, has_cache);
  auto kern = extra ? frnn_fwd_reg_kernel<CELL, KT, LOCAL, NB, DENSE, true> : frnn_fwd_reg_kernel<CELL, KT, LOCAL, NB, DENSE, false>;
  FwdParams q = p;
  q.C = (p.D + U - 1) / U;
  const long long groups = static_cast<long long>(p.N) * reg_batch_tiles(p.B, ROWS);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(groups * q.C));
  cfg.blockDim = dim3(static_cast<unsigned>(Cfg::THREADS));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(q.C);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = LOCAL ? 0 : 1;
  if constexpr (KT == 4 && NB == 1 && !DENSE && CELL != kElman) {
    // Heads of 64 units: three CTAs of nine warps an SM within 72 registers cost a step 3 to 9 %, but hold groups that would need 16 rows. B304
    // T64 N4, us, 16 rows / three CTAs: LSTM 58 / 52, sLSTM 81 / 66, GRU 52 / 48. The sLSTM with fp32 Wx, 82 / 74, stays with 16 rows.
    const int two = reg_capacity(reinterpret_cast<const void*>(kern), cfg, q.C);
    if (two >= 0 && groups > two && (CELL != kSLSTM || wx_bf16)) return launch_fwd_reg<CELL, KT, LOCAL, NB, true>(p, wx, wx_bf16, stream, ask, rival_groups);
  }
  if constexpr (KT == 12 && NB == 1 && !DENSE && CELL != kElman) {
    // Heads of 144 to 192 units: two CTAs an SM within 96 registers, where wider groups would not be fewer. B8 T48, us, tcgen05 / these: N34
    // D144 LSTM 105 / 43, sLSTM 116 / 50, GRU 61 / 40; N24 D192 LSTM 65 / 43, GRU 61 / 40. Heads that fit with one CTA an SM have 118 to 124 registers.
    const int one = reg_capacity(reinterpret_cast<const void*>(kern), cfg, q.C);
    if (one >= 0 && groups > one && p.B <= kRegRows) return launch_fwd_reg<CELL, KT, LOCAL, NB, true>(p, wx, wx_bf16, stream, ask, rival_groups);
  }
  // whether the call is taken at all comes first: one that is not pays for nothing else
  const int rc = reg_room(reinterpret_cast<const void*>(kern), cfg, q.C, groups, rival_groups, p.D);
  if (rc != 0 || ask) return rc != 0 ? rc : kRegTaken;
  CUtensorMap map, hist_map, cache_map, hbf_map;
  const uint64_t nd = static_cast<uint64_t>(p.N) * p.D, T = p.T, Tt = p.T_total;
  const int end = p.t0 + p.T;  // steps past the call's own are neither read nor written
  const auto tile_map = [&](CUtensorMap* m, const void* base, int bytes, int planes, int steps_end, uint64_t bs, uint64_t ps, uint64_t ss) {
    return reg_tile_map(m, base, bytes, p.D, p.N, p.B, planes, steps_end, bs, ps, ss, planes, CHUNK, ROWS, steps);
  };
  if (tile_map(&map, wx, es, CT::GW, end, Tt * CT::GW * nd, nd, CT::GW * nd) != 0) return -4;
  hist_map = cache_map = hbf_map = map;  // valid maps where a stream is not written
  if (hist_states > 0 && tile_map(&hist_map, p.history, hes, hist_states, end, Tt * nd, p.B * Tt * nd, nd) != 0) return -4;
  if (has_cache && tile_map(&cache_map, p.cache, CT::CES, CT::GC, p.T, T * CT::GC * nd, nd, CT::GC * nd) != 0) return -4;
  if (p.hbf != nullptr && tile_map(&hbf_map, p.hbf + nd, 2, 1, p.T, (T + 1) * nd, nd, nd) != 0) return -4;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, q, map, hist_map, cache_map, hbf_map, wx_bf16, steps, hist_states));
}

template <int CELL, int KT, bool LOCAL>
int launch_fwd_reg_rows(const FwdParams& p, const void* wx, int wx_bf16, cudaStream_t s, int rows, bool ask) {
  const long long rivals = LOCAL ? static_cast<long long>(p.N) * reg_batch_tiles(p.B, 16) : 0;
  if (rows == kRegRows) return launch_fwd_reg<CELL, KT, LOCAL, 1>(p, wx, wx_bf16, s, ask, rivals);
  // More rows per group: 13 to 14 cycles of a scheduler per mma and column tile, while a tcgen05.mma costs the same for 16 rows as for 8
  // and its kernel has two CTAs of up to 448 units on an SM. T48 N1 - 4, us, against that kernel: 16 rows LSTM B64 D448 105 / 102, D512
  // 120 / 222; 24 rows B96 D256 344 / 411 (T256), B256 D288 108 / 99, B64 D384 116 / 108. The Elman cell has half the tiles: D512 153 / 327.
  // Of 16-row groups of the sLSTM from 480 units on, a training call with bf16 Wx loses to tcgen05 groups that run in one wave, and wins
  // where these need a second one: B112 T48 D512 151 / 133 us, B64 144 / 221 (fp32 Wx 117 / 134, inference 111 / 123).
  if (rows == 2 * kRegRows) {
    if (CELL != kElman && p.D > 384 && p.D <= 448) return kRegNoRoom;
    if constexpr (CELL == kSLSTM && KT == 32) {
      if (p.D >= 480 && wx_bf16 && p.cache != nullptr && reg_rival(false, CELL, wx_bf16, p.N, p.B, p.D).waves == 1) return kRegNoRoom;
    }
    return launch_fwd_reg<CELL, KT, LOCAL, 2>(p, wx, wx_bf16, s, ask, rivals);
  }
  if constexpr (KT == 12 || KT == 16 || (CELL == kElman && KT > 16)) return launch_fwd_reg<CELL, KT, LOCAL, 3>(p, wx, wx_bf16, s, ask);
  return kRegNoRoom;
}

}  // namespace

template <int CELL>
int launch_fwd_reg_cell(const FwdParams& p, const void* wx, int wx_bf16, cudaStream_t s, int rows, bool ask) {
  switch (reg_k_tiles(p.D)) {
    case 1: return launch_fwd_reg_rows<CELL, 1, true>(p, wx, wx_bf16, s, rows, ask);
    case 2: return launch_fwd_reg_rows<CELL, 2, true>(p, wx, wx_bf16, s, rows, ask);
    case 3: return launch_fwd_reg_rows<CELL, 3, true>(p, wx, wx_bf16, s, rows, ask);
    case 4: return launch_fwd_reg_rows<CELL, 4, false>(p, wx, wx_bf16, s, rows, ask);
    case 6: return launch_fwd_reg_rows<CELL, 6, false>(p, wx, wx_bf16, s, rows, ask);
    case 8: return launch_fwd_reg_rows<CELL, 8, false>(p, wx, wx_bf16, s, rows, ask);
    case 10:
    case 12: return launch_fwd_reg_rows<CELL, 12, false>(p, wx, wx_bf16, s, rows, ask);
    case 14:
    case 16: return launch_fwd_reg_rows<CELL, 16, false>(p, wx, wx_bf16, s, rows, ask);
    case 20:
    case 24: return launch_fwd_reg_rows<CELL, 24, false>(p, wx, wx_bf16, s, rows, ask);
    case 28:
    case 32: return launch_fwd_reg_rows<CELL, 32, false>(p, wx, wx_bf16, s, rows, ask);
    default: return -2;
  }
}

}  // namespace frnn
