// Reverse-time recurrence of wide heads with R in the register file (see recurrent_wide_fwd.cuh, recurrent_reg_bwd.cuh).
//
// The decomposition is that of recurrent_bwd_ksplit.cu: a group is D/128 tiles of 128 units p times KS chunks of the K = GR * D gate
// rows, the KS CTAs of a tile are a cluster, each owns 128 / KS units. Warp w of a CTA has the fragments of R[k, p]^T for the units
// 16w .. 16w + 15 of the tile and the CTA's chunk of k. Per step
//   1. the owner warps add the KS partial dh_t of their items (in their order: the sums are those of the tensor-memory kernel, bit for
//      bit), run the cell backward and store the words of round_bf16(dG_t) (two batch rows of a gate row) to the slot of the step,
//   2. all warps fetch the packets (8 batch rows of a gate row) of their chunk,
//   3. multiply, and send the partial dh_{t-1} to the CTA that owns the unit (st.async, two batch rows of a unit).
// Slots, refills and fences as in recurrent_wide_fwd.cuh.
//
// Bound: the serial chain of a step, two hops of it: LSTM B16 N1 D768, cycles: dG_t of the other CTAs polled 1052, mma and scatter 1027,
// tiles read, partial sums awaited and added 689, cell and publication 399. us per step of the tensor-memory kernel and here: there
// 2.48 / 1.74, B4 2.26 / 1.67; GRU D768 2.22 / 1.66; LSTM B8 D896 2.62 / 2.00, D1024 2.78 / 2.17; Elman B16 D1024 2.11 / 1.48.
#pragma once

#include <type_traits>

#include "recurrent_reg.cuh"

namespace frnn {

namespace {

// History planes the cell's derivative reads: [first, first + count).
template <int CELL> struct WideHistPlanes;
template <> struct WideHistPlanes<kLSTM> { static constexpr int first = 1, count = 1; };
template <> struct WideHistPlanes<kSLSTM> { static constexpr int first = 1, count = 3; };
template <> struct WideHistPlanes<kGRU> { static constexpr int first = 0, count = 1; };
template <> struct WideHistPlanes<kElman> { static constexpr int first = 0, count = 1; };

template <int CELL, int KS, int NB, int KT>
struct BwdWideCfg {
  using CT = CellTraits<CELL>;
  static constexpr int UO = 128 / KS, GROUPS = UO * NB / 4;        // units owned; groups of 4 units x 8 rows (an item per lane)
  static constexpr int OWNERS = GROUPS < 8 ? GROUPS : 8, IPT = GROUPS / OWNERS;
  static constexpr int ROWS = NB * kRegRows, CHUNK = UO < 32 ? UO : 32, CHUNKS = UO / CHUNK, THREADS = 9 * 32;
  static constexpr int HALF = KT * 256, DG = NB * HALF;            // operand: [column tile][k][8 batch rows]
  static constexpr int PART_TILE = UO * 32, PART = KS * NB * PART_TILE;  // one parity: [source][column tile][unit][8 batch rows] fp32
  static constexpr int FIXED = reg_round_1k(2 * DG + 2 * PART);
  static constexpr int GCL = CELL == kElman ? 0 : CT::GC;
  static constexpr int HP = WideHistPlanes<CELL>::first, HS = WideHistPlanes<CELL>::count;
  static constexpr int PLANE2 = ROWS * CHUNK * 2, PLANE4 = ROWS * CHUNK * 4, PLANEC = ROWS * CHUNK * CT::CES;
  static_assert(2 * PART >= NB * 8 * CT::GB * UO * 4, "the bias sums of the last step fit the buffers of the partial sums");
};

template <int CELL, int KS, int NB, int KT, bool EXTRA>
__global__ void __launch_bounds__(BwdWideCfg<CELL, KS, NB, KT>::THREADS, 1)
frnn_bwd_wide_kernel(const BwdParams p, const float* history, const float* initial, const __grid_constant__ CUtensorMap cache_map,
                     const __grid_constant__ CUtensorMap hist_map, const __grid_constant__ CUtensorMap dhist_map,
                     const __grid_constant__ CUtensorMap dgr_map, const __grid_constant__ CUtensorMap dwx_map, const int wx_bf16,
                     const int own_dwx, const int ring_steps, const int xg_slots) {
  using Cfg = BwdWideCfg<CELL, KS, NB, KT>;
  using CT = CellTraits<CELL>;
  constexpr int S = CT::S, UO = Cfg::UO, CHUNK = Cfg::CHUNK, ROWS = Cfg::ROWS, OWNERS = Cfg::OWNERS, IPT = Cfg::IPT, GCL = Cfg::GCL,
                HP = Cfg::HP, HS = Cfg::HS, kPlane2 = Cfg::PLANE2, kPlane4 = Cfg::PLANE4;

  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t s_part_bar[2];
  __shared__ int s_gave_up;  // a compute warp of this CTA has stopped waiting
  __shared__ __align__(8) uint64_t s_full[kRegSlots];
  __shared__ __align__(8) uint64_t s_out_full[kRegSlots];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane >> 2, c = lane & 3, hi = lane >> 4, uq = q & 3;
  const long long t_entry = clock64();
  const int D = p.D, N = p.N, T = p.T, B = p.B, PT = D / 128, K = CT::GR * D, Kc = K / KS;
  const int ks = static_cast<int>(blockIdx.x % KS);  // == rank inside the cluster
  const int pt = static_cast<int>(blockIdx.x / KS % PT), gid = static_cast<int>(blockIdx.x / (KS * PT));
  const int n = gid % N, btile = gid / N, b0 = btile * ROWS;
  const int u0 = pt * 128 + ks * UO;  // first owned unit
  uint8_t* const dgbuf = smem;
  uint8_t* const part = smem + 2 * Cfg::DG;
  uint8_t* const stages = smem + Cfg::FIXED;
  // a transfer of inputs: per chunk of units the cache, the states of step t - 1, the external gradient, each from a multiple of 1 KB
  const int region_h = reg_round_1k(ring_steps * GCL * Cfg::PLANEC), region_d = region_h + reg_round_1k(ring_steps * HS * kPlane4);
  const int in_chunk = region_d + reg_round_1k(ring_steps * S * kPlane4), stage_bytes = Cfg::CHUNKS * in_chunk;
  uint8_t* const outs = stages + kRegSlots * stage_bytes;
  const int dwx_bytes = own_dwx ? CT::GW * (wx_bf16 ? kPlane2 : kPlane4) : 0;
  const int region_g = reg_round_1k(ring_steps * dwx_bytes), out_chunk = region_g + reg_round_1k(ring_steps * CT::GR * kPlane2);
  const int out_slot = Cfg::CHUNKS * out_chunk;
  const uint32_t slot_bytes = static_cast<uint32_t>(ROWS) * K * 2u;
  uint8_t* const xg = p.xg_data + static_cast<size_t>(gid) * xg_slots * slot_bytes;
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
      mbar_init(smem_u32(&s_out_full[i]), OWNERS);
    }
    s_gave_up = 0;
    fence_mbar_init();
  }
  for (int i = tid; i < 2 * Cfg::DG / 16; i += blockDim.x) reinterpret_cast<uint4*>(dgbuf)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  if (tid == 0) {
    mbar_arrive_expect_tx(smem_u32(&s_part_bar[1]), Cfg::PART);              // iteration 1 (the last one if T == 1)
    if (T >= 2) mbar_arrive_expect_tx(smem_u32(&s_part_bar[0]), Cfg::PART);  // iteration 2
  }

  if (warp == 8) {
    // ---------------- I/O warp: tiles in, staged outputs out ----------------
    cluster_sync_all();
    if (lane == 0) {
      auto fill = [&](int t0, int s) {  // see recurrent_reg_bwd.cuh
        const uint32_t bar = smem_u32(&s_full[s]);
        mbar_arrive_expect_tx(bar, static_cast<uint32_t>(Cfg::CHUNKS * ring_steps * (GCL * Cfg::PLANEC + (HS + S) * kPlane4)));
#pragma unroll
        for (int i = 0; i < Cfg::CHUNKS; ++i) {
          const uint32_t dst = smem_u32(stages + s * stage_bytes + i * in_chunk);
          const int x = u0 + i * CHUNK;
          if (GCL > 0) tma_load_5d(dst, &cache_map, bar, x, n, b0, 0, t0);
          tma_load_5d(dst + region_h, &hist_map, bar, x, n, b0, HP, t0 - 1);
          tma_load_5d(dst + region_d, &dhist_map, bar, x, n, b0, 0, t0);
        }
      };
      const int last = (T - 1) / ring_steps * ring_steps;
      for (int i = 0; i < kRegSlots && last - i * ring_steps >= 0; ++i) fill(last - i * ring_steps, i);
      int slot = 0;
      uint32_t phase = 0;
      auto staged = [&](int step) -> bool {  // as in recurrent_reg_fwd.cuh
        const uint32_t bar = smem_u32(&s_out_full[slot]);
        for (int fast = 0; fast < 64; ++fast)
          if (mbar_try_wait(bar, phase)) return true;
        if (jitter != 0u) jitter_stall(jitter, 32u, static_cast<uint32_t>(step));
        return mbar_wait_bounded<false>(bar, phase, 2 * limit, abort_flag);
      };
      for (int t0 = last; t0 >= 0; t0 -= ring_steps) {
        if (!staged(T - 1 - t0)) {
          reg_report(p.err, kErrWaitEmpty, T - 1 - t0);
          break;
        }
        // A warp that gave up on a wait sets the flag before it stages: see recurrent_reg_fwd.cuh.
        if (*reinterpret_cast<volatile int*>(&s_gave_up) != 0) break;
#pragma unroll
        for (int i = 0; i < Cfg::CHUNKS; ++i) {
          const uint32_t src = smem_u32(outs + slot * out_slot + i * out_chunk);
          const int x = u0 + i * CHUNK;
          if (own_dwx) tma_store_5d(&dwx_map, src, x, n, b0, 0, t0);
          tma_store_5d(&dgr_map, src + region_g, x, n, b0, 0, t0);
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
    // A fragments of R[chunk, tile]^T: 8x8 blocks of R are loaded as they lie (gate rows x units p) and transposed in the warp.
    uint32_t a[KT][4];
#pragma unroll
    for (int j = 0; j < KT; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int k = j * 16 + 8 * (r >> 1) + q, kg = ks * Kc + k, g = kg / D, o = kg - g * D;
        const int pcol = pt * 128 + warp * 16 + 8 * (r & 1) + 2 * c;
        uint32_t v = 0u;
        if (k < Kc) v = __ldg(reinterpret_cast<const uint32_t*>(p.R + ((static_cast<size_t>(g) * N + n) * D + o) * D + pcol));
        a[j][r] = movmatrix_trans(v);
      }

    // items of a thread of an owner warp: one unit of one batch row each
    const size_t ND = static_cast<size_t>(N) * D, BND = static_cast<size_t>(B) * ND, sBTND = static_cast<size_t>(T) * BND;
    const bool owner = warp < OWNERS;
    const int row = 2 * c + hi;  // row of the column tile
    auto item_tile = [&](int i) { return (warp + OWNERS * i) / (UO / 4); };
    auto item_unit = [&](int i) { return (warp + OWNERS * i) % (UO / 4) * 4 + uq; };
    bool act[IPT];
    float dcar[S][IPT], dbacc[CT::GB][IPT], sn[HS][IPT];
    uint32_t off2[IPT], off4[IPT], in_at[IPT], out_at[IPT], part_src[IPT], word_at[IPT];
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      const int ul = item_unit(i), tile = item_tile(i), d = u0 + ul, b = b0 + tile * 8 + row;
      act[i] = owner && b < B;
      const size_t item = static_cast<size_t>(b) * ND + static_cast<size_t>(n) * D + d;
#pragma unroll
      for (int g = 0; g < CT::GB; ++g) dbacc[g][i] = 0.0f;
#pragma unroll
      for (int k = 0; k < S; ++k) dcar[k][i] = act[i] ? p.d_carry[k * BND + item] : 0.0f;
#pragma unroll
      for (int k = 0; k < HS; ++k)
        sn[k][i] = act[i] ? history[(HP + k) * sBTND + (static_cast<size_t>(b) * T + T - 1) * ND + static_cast<size_t>(n) * D + d] : 0.0f;
      off2[i] = reg_tile_offset<2, CHUNK>(tile * 8 + row, ul % CHUNK);
      off4[i] = reg_tile_offset<4, CHUNK>(tile * 8 + row, ul % CHUNK);
      in_at[i] = static_cast<uint32_t>(ul / CHUNK * in_chunk);
      out_at[i] = static_cast<uint32_t>(ul / CHUNK * out_chunk);
      part_src[i] = smem_u32(part) + static_cast<uint32_t>(tile * Cfg::PART_TILE + ul * 32 + row * 4);
      word_at[i] = static_cast<uint32_t>(tile * K + d + (CT::GR > 1 ? hi * D : 0)) * 16 + c * 4;  // of the gate that the lane publishes
    }
    const bool v1 = p.slstm_v1 != 0, zero_first = p.slstm_zero_first != 0, cut = p.cut_recurrent != 0, clip_on = p.grad_clip > 0.0f;
    const float grad_clip = p.grad_clip;
    // where the partial sums of this warp's 16 units go
    const uint32_t delta = map_to_cta(smem_u32(smem), static_cast<uint32_t>(16 * warp / UO)) - smem_u32(smem);
    const uint32_t part_dst = smem_u32(part) + static_cast<uint32_t>(ks * NB * Cfg::PART_TILE + (16 * warp % UO + q) * 32 + c * 8);
    constexpr int J = (NB * KT * 16 + 255) / 256;  // packets this thread fetches
    const int packets = NB * Kc;
    bool dead = false;  // warp-uniform: after a failed wait the warp walks on without waiting
    auto give_up = [&](int code, int it) {
      if (lane == 0) reg_report(p.err, code, it);
      dead = true;
      *reinterpret_cast<volatile int*>(&s_gave_up) = 1;
    };
    cluster_sync_all();
    if (prof) p.err[20] = static_cast<int>(clock64() - t_entry);

    // Partial sums of iteration `it`, added in the order of their sources.
    auto add_parts = [&](int it, float (&dsum)[IPT]) {
#pragma unroll
      for (int i = 0; i < IPT; ++i) {
        float v[KS];
#pragma unroll
        for (int s = 0; s < KS; ++s) v[s] = lds_f32(part_src[i] + (it & 1) * Cfg::PART + s * (NB * Cfg::PART_TILE));
#pragma unroll
        for (int s = 0; s < KS; ++s) dsum[i] += v[s];
      }
    };
    // The steps, compiled without the options and hooks of a call, with the options, and with both.
    auto run = [&](auto mode_tag) {
      constexpr bool hook = decltype(mode_tag)::value == kRegHooks, any = decltype(mode_tag)::value != kRegPlain;
      long long pc[6] = {0, 0, 0, 0, 0, 0};
      auto clock = [&]() -> long long { return hook && prof ? clock64() : 0; };
      auto wait_parts = [&](int it) {
        if (!dead && !mbar_wait_warp<true>(smem_u32(&s_part_bar[it & 1]), ((it - 1) >> 1) & 1, limit, abort_flag)) give_up(kErrWaitPart, it);
      };
      int slot = 0, it = 0;
      uint32_t in_phase = 0;
      for (int t0 = (T - 1) / ring_steps * ring_steps; t0 >= 0; t0 -= ring_steps) {
        if (owner && !dead && !mbar_wait_warp<false>(smem_u32(&s_full[slot]), in_phase, limit, abort_flag)) give_up(kErrWaitWx, it);
        const int first = T - 1 - it - t0;  // step of the transfer it begins with, counting down
        const uint32_t in = smem_u32(stages) + slot * stage_bytes, out = smem_u32(outs) + slot * out_slot;
        for (int t = t0 + first; t >= t0; --t, ++it) {
          if (hook && jitter != 0u) { jitter_stall(jitter, static_cast<uint32_t>(warp), static_cast<uint32_t>(it)); __syncwarp(); }
          const long long c1 = clock();
          long long c2 = c1, c3 = c1;
          if (owner) {
            const int j = t - t0;
            float cache[CT::GC][IPT], sp[HS][IPT], dh[S][IPT], ds[S][IPT];
#pragma unroll
            for (int i = 0; i < IPT; ++i) {
              const uint32_t at = in + in_at[i];
#pragma unroll
              for (int g = 0; g < GCL; ++g) {
                const uint32_t x = at + (j * GCL + g) * Cfg::PLANEC;
                if constexpr (CT::CES == 2) cache[g][i] = __half2float(__ushort_as_half(static_cast<unsigned short>(lds_u16(x + off2[i]))));
                else cache[g][i] = lds_f32(x + off4[i]);
              }
#pragma unroll
              for (int k = 0; k < HS; ++k) sp[k][i] = lds_f32(at + region_h + (j * HS + k) * kPlane4 + off4[i]);
#pragma unroll
              for (int k = 0; k < S; ++k) dh[k][i] = lds_f32(at + region_d + (j * S + k) * kPlane4 + off4[i]);
              if (t == 0 && act[i]) {
#pragma unroll
                for (int k = 0; k < HS; ++k)
                  sp[k][i] = initial[(HP + k) * BND + static_cast<size_t>(b0 + item_tile(i) * 8 + row) * ND + static_cast<size_t>(n) * D + u0 + item_unit(i)];
              }
#pragma unroll
              for (int k = 0; k < S; ++k) ds[k][i] = dcar[k][i] + dh[k][i];
            }
            if (it >= 1) {
              wait_parts(it);
              if (!(any && cut)) add_parts(it, ds[0]);
            }
            if (any && clip_on && it >= 1) {
              // the gradient carried into h_t from step t + 1 (total minus the external part) is complete here: clip it
#pragma unroll
              for (int i = 0; i < IPT; ++i) ds[0][i] = clip_sym(ds[0][i] - dh[0][i], grad_clip) + dh[0][i];
            }
            c2 = clock();
            const bool take_i = CELL == kSLSTM && t == 0 && zero_first;
            const bool publish = !(hook && (dead || it >= mute_from));
            uint8_t* const xg_now = xg + static_cast<size_t>(it % kWideSlots) * slot_bytes;
            uint8_t* const xg_ahead = xg + static_cast<size_t>((it + kWideSlots / 2) % kWideSlots) * slot_bytes;
            const bool refill = it + kWideSlots / 2 < T && it + kWideSlots / 2 >= xg_slots;
#pragma unroll
            for (int i = 0; i < IPT; ++i) {
              float cj[CT::GC], snj[S], spj[S], dsj[S], gr[CT::GR], gw[CT::GW], gb[CT::GB];
#pragma unroll
              for (int g = 0; g < GCL; ++g) cj[g] = cache[g][i];
#pragma unroll
              for (int k = 0; k < S; ++k) {
                snj[k] = k >= HP && k < HP + HS ? sn[k >= HP ? k - HP : 0][i] : 0.0f;
                spj[k] = k >= HP && k < HP + HS ? sp[k >= HP ? k - HP : 0][i] : 0.0f;
                dsj[k] = ds[k][i];
              }
              cell_backward<CELL>(cj, spj, snj, dsj, gr, gw, gb, take_i, any && v1);
              // Rows past the batch hold zeros: so do their gradients, but where the cell divides.
              constexpr bool drop = CELL == kSLSTM;
#pragma unroll
              for (int k = 0; k < S; ++k) dcar[k][i] = !drop || act[i] ? dsj[k] : 0.0f;
#pragma unroll
              for (int g = 0; g < CT::GR; ++g) gr[g] = !drop || act[i] ? gr[g] : 0.0f;
#pragma unroll
              for (int g = 0; g < CT::GW; ++g) gw[g] = !drop || act[i] ? gw[g] : 0.0f;
#pragma unroll
              for (int k = 0; k < HS; ++k) sn[k][i] = sp[k][i];
              // Words of dG_t, two gates at a time: the lanes 16 apart have the rows 2c and 2c + 1 and a gate's word each.
              uint32_t dgp[CT::GR];
#pragma unroll
              for (int g = 0; g < CT::GR; ++g) dgp[g] = bf16_bits(gr[g]);
#pragma unroll
              for (int g = 0; g < CT::GR; g += 2) {
                const bool two = g + 1 < CT::GR;
                const uint32_t second = dgp[two ? g + 1 : g], other = __shfl_xor_sync(0xffffffffu, hi ? dgp[g] : second, 16);
                const uint32_t w = xg_clean(hi ? other | second << 16 : dgp[g] | other << 16);
                const size_t at = word_at[i] + static_cast<size_t>(g * D) * 16;
                if (publish && !dead && (two || !hi)) st_relaxed_gpu_u32(xg_now + at, w);
              }
              if (publish && !dead && refill) {
#pragma unroll
                for (int g = 0; g < CT::GR; g += 2)
                  if (g + 1 < CT::GR || !hi) st_relaxed_gpu_u32(xg_ahead + word_at[i] + static_cast<size_t>(g * D) * 16, kXgFill);
              }
              // outputs and bias sums, while dG_t is on its way
#pragma unroll
              for (int g = 0; g < CT::GR; ++g) sts_u16(out + out_at[i] + region_g + (j * CT::GR + g) * kPlane2 + off2[i], dgp[g]);
              if (own_dwx) {
#pragma unroll
                for (int g = 0; g < CT::GW; ++g) {
                  const uint32_t at = out + out_at[i] + j * dwx_bytes;
                  if (wx_bf16) sts_u16(at + g * kPlane2 + off2[i], bf16_bits(gw[g]));
                  else sts_f32(at + g * kPlane4 + off4[i], gw[g]);
                }
              }
#pragma unroll
              for (int g = 0; g < CT::GB; ++g) dbacc[g][i] += CELL != kGRU ? gw[g] : (g == 0 ? gr[0] : gw[g > 0 ? g - 1 : 0]);  // as cell_backward's gb
            }
            // this parity's partial sums were complete at the wait: armed for iteration it + 2
            if (tid == 0 && !dead && it >= 1 && it + 2 <= T) mbar_arrive_expect_tx(smem_u32(&s_part_bar[it & 1]), Cfg::PART);
            c3 = clock();
          }
          // this CTA's chunk of dG_t -> operand buffer of this parity
          {
            const uint8_t* const from = xg + static_cast<size_t>(it % kWideSlots) * slot_bytes + static_cast<size_t>(ks) * Kc * 16;
            const uint32_t dst = smem_u32(dgbuf) + (it & 1) * Cfg::DG;
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
                if ((pend >> j) & 1u) v[j] = ld_relaxed_gpu_v4(from + static_cast<size_t>(half * K + k) * 16);
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
            if (__any_sync(0xffffffffu, pend != 0u)) give_up(kErrWaitDg, it);
            if ((it & (kWideFence - 1)) == kWideFence - 1) fence_acq_rel_gpu();
            asm volatile("bar.sync 1, 256;" ::: "memory");
          }
          const long long c4 = clock();
          const int nb = (it + 1) & 1;
          {
            float acc[NB][4];
#pragma unroll
            for (int e = 0; e < NB; ++e)
#pragma unroll
              for (int r = 0; r < 4; ++r) acc[e][r] = 0.0f;
            const uint32_t db = smem_u32(dgbuf) + (it & 1) * Cfg::DG + lane * 16;
#pragma unroll
            for (int k2 = 0; k2 < KT / 2; ++k2) {
              uint32_t bf[NB][4];
#pragma unroll
              for (int e = 0; e < NB; ++e) ldsm_x4_trans(db + e * Cfg::HALF + k2 * 512, bf[e]);
#pragma unroll
              for (int e = 0; e < NB; ++e) mma_bf16_16816(acc[e], a[2 * k2], bf[e][0], bf[e][1]);
#pragma unroll
              for (int e = 0; e < NB; ++e) mma_bf16_16816(acc[e], a[2 * k2 + 1], bf[e][2], bf[e][3]);
            }
            const uint32_t bar = smem_u32(&s_part_bar[nb]) + delta;
            if (!dead) {
#pragma unroll
              for (int e = 0; e < NB; ++e) {
                const uint32_t dst = part_dst + delta + nb * Cfg::PART + e * Cfg::PART_TILE;
                st_async_v2_b32(dst, __float_as_uint(acc[e][0]), __float_as_uint(acc[e][1]), bar);
                st_async_v2_b32(dst + 8 * 32, __float_as_uint(acc[e][2]), __float_as_uint(acc[e][3]), bar);
              }
            }
          }
          const long long c5 = clock();
          if (hook && prof) {
            pc[0] += c5 - c1; pc[1] += c2 - c1; pc[2] += c3 - c2; pc[3] += c4 - c3; pc[4] += c5 - c4;
          }
        }
        if (owner) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&s_out_full[slot]));
        }
        if (++slot == kRegSlots) { slot = 0; in_phase ^= 1u; }
      }
      if (owner) {
        wait_parts(T);
        if (!(any && cut)) add_parts(T, dcar[0]);
      }
      if (hook && prof) {
        p.err[15] = static_cast<int>(pc[0]);  // the whole step
        p.err[9] = static_cast<int>(pc[1]);   // tiles read, wait for the partial sums, their sum
        p.err[10] = static_cast<int>(pc[2]);  // cell, publication, outputs staged
        p.err[11] = static_cast<int>(pc[3]);  // dG of the other CTAs, barrier
        p.err[12] = static_cast<int>(pc[4]);  // mma and scatter
      }
    };
    if (hooks || (!EXTRA && (cut || clip_on || v1))) run(std::integral_constant<int, kRegHooks>{});
    else run(std::integral_constant<int, EXTRA ? kRegAny : kRegPlain>{});
    // bias gradient of the batch rows of the group, added in their order: through the buffers of the partial sums, which the last wait
    // of every owner warp left
    asm volatile("bar.sync 1, 256;" ::: "memory");
    float* const sums = reinterpret_cast<float*>(part);
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      const int ul = item_unit(i), r8 = item_tile(i) * 8 + row;
      if (act[i]) {
#pragma unroll
        for (int k = 0; k < S; ++k)
          p.d_initial[k * BND + static_cast<size_t>(b0 + r8) * ND + static_cast<size_t>(n) * D + u0 + ul] = dcar[k][i];
      }
      if (owner) {
#pragma unroll
        for (int g = 0; g < CT::GB; ++g) sums[(r8 * CT::GB + g) * UO + ul] = dbacc[g][i];
      }
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    for (int i = tid; i < CT::GB * UO; i += 256) {
      float v = 0.0f;
      for (int r = 0; r < ROWS && b0 + r < B; ++r) v += sums[r * CT::GB * UO + i];
      p.db_part[((static_cast<size_t>(btile) * CT::GB + i / UO) * N + n) * D + u0 + i % UO] = v;
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
int launch_bwd_wide(const BwdParams& p, const void* cache, const float* history, const float* initial, const float* d_history,
                    int wx_bf16, cudaStream_t stream, bool ask) {
  using Cfg = BwdWideCfg<CELL, KS, NB, KT>;
  using CT = CellTraits<CELL>;
  const bool own_dwx = !wx_bf16 || CELL == kGRU || p.dwx != static_cast<void*>(p.dgr);
  const auto bytes = [&](int st) {
    return Cfg::FIXED + kRegSlots * Cfg::CHUNKS *
                            (reg_round_1k(st * Cfg::GCL * Cfg::PLANEC) + reg_round_1k(st * Cfg::HS * Cfg::PLANE4) + reg_round_1k(st * CT::S * Cfg::PLANE4) +
                             reg_round_1k(own_dwx ? st * CT::GW * (wx_bf16 ? Cfg::PLANE2 : Cfg::PLANE4) : 0) + reg_round_1k(st * CT::GR * Cfg::PLANE2));
  };
  int steps = 4;
  while (steps > 1 && bytes(steps) > kRegSmemLimit) --steps;
  const int smem = bytes(steps);
  if (smem > kRegSmemLimit) return kRegNoRoom;
  if (((reinterpret_cast<uintptr_t>(p.dwx) | reinterpret_cast<uintptr_t>(p.dgr)) & 15u) != 0) return kRegNoRoom;  // off the grid of bulk stores
  auto kern = reg_extra(p) ? frnn_bwd_wide_kernel<CELL, KS, NB, KT, true> : frnn_bwd_wide_kernel<CELL, KS, NB, KT, false>;
  const int D = p.D, N = p.N, B = p.B;
  const long long groups = static_cast<long long>(N) * reg_batch_tiles(B, Cfg::ROWS), clusters = groups * (D / 128);
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
  const int rc = reg_room(reinterpret_cast<const void*>(kern), cfg, KS, clusters, 0, D);
  if (rc != 0 || ask) return rc != 0 ? rc : kRegTaken;
  CUtensorMap cache_map, hist_map, dhist_map, dgr_map, dwx_map;
  const uint64_t nd = static_cast<uint64_t>(N) * D, uT = p.T, uB = p.B;
  const auto map = [&](CUtensorMap* m, const void* base, int es, int planes, uint64_t bs, uint64_t ps, uint64_t ss, int box_planes) {
    return reg_tile_map(m, base, es, D, N, B, planes, p.T, bs, ps, ss, box_planes, Cfg::CHUNK, Cfg::ROWS, steps);
  };
  if (map(&hist_map, history, 4, CT::S, uT * nd, uB * uT * nd, nd, Cfg::HS) != 0 ||
      map(&dhist_map, d_history, 4, CT::S, uT * nd, uB * uT * nd, nd, CT::S) != 0 ||
      map(&dgr_map, p.dgr, 2, CT::GR, uT * CT::GR * nd, nd, CT::GR * nd, CT::GR) != 0)
    return -4;
  cache_map = hist_map;  // Elman has no cache: a valid map that is never used
  if (Cfg::GCL > 0 && map(&cache_map, cache, CT::CES, CT::GC, uT * CT::GC * nd, nd, CT::GC * nd, CT::GC) != 0) return -4;
  dwx_map = dgr_map;
  if (own_dwx && map(&dwx_map, p.dwx, wx_bf16 ? 2 : 4, CT::GW, uT * CT::GW * nd, nd, CT::GW * nd, CT::GW) != 0) return -4;
  const int slots = wide_slots(p.T);
  const cudaError_t me = cudaMemsetAsync(p.xg_data, 0xff, static_cast<size_t>(groups) * slots * Cfg::ROWS * CT::GR * D * 2, stream);
  if (me != cudaSuccess) return static_cast<int>(me);
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, p, history, initial, cache_map, hist_map, dhist_map, dgr_map, dwx_map, wx_bf16,
                                             own_dwx ? 1 : 0, steps, slots));
}

struct BwdWideCall {
  const BwdParams& p;
  const void* cache;
  const float *history, *initial, *d_history;
  int wx_bf16;
  cudaStream_t stream;
  bool ask;
};

template <int CELL, int KS, int NB>
int launch_bwd_wide_k(const BwdWideCall& v) {
  const int kc = CellTraits<CELL>::GR * v.p.D / KS;
  if (kc % 16 != 0) return kRegNoRoom;
  const int kt = kc / 16;
  const auto go = [&](auto bound) {
    return launch_bwd_wide<CELL, KS, NB, decltype(bound)::value>(v.p, v.cache, v.history, v.initial, v.d_history, v.wx_bf16, v.stream, v.ask);
  };
  if (kt <= 12) return go(std::integral_constant<int, 12>{});
  if (kt <= 18) return go(std::integral_constant<int, 18>{});
  if (kt <= 24) return go(std::integral_constant<int, 24>{});
  if (kt <= 28) return go(std::integral_constant<int, 28>{});
  // 128 of the 168 registers are fragments: B16 N1 D1024 (16 rows a group) LSTM 3.34 / 3.12 us per step, sLSTM 3.61 / 3.64
  if (NB == 2 && CELL == kSLSTM) return kRegNoRoom;
  if (kt <= 32) return go(std::integral_constant<int, 32>{});
  return kRegNoRoom;
}

}  // namespace

// The call of a plan with `ksplit` CTAs per tile of 128 units and `rows` batch rows per group, or kRegNoRoom (its fragments do not fit
// the registers, outputs off the 16-byte grid, clusters that do not fit). Fills the exchange slots itself. `ask`: only say whether (kRegTaken).
template <int CELL>
int launch_bwd_wide_cell(const BwdParams& p, const void* cache, const float* history, const float* initial, const float* d_history,
                         int wx_bf16, int rows, int ksplit, cudaStream_t s, bool ask) {
  const BwdWideCall v{p, cache, history, initial, d_history, wx_bf16, s, ask};
  if (ksplit == 8) return rows == 8 ? launch_bwd_wide_k<CELL, 8, 1>(v) : launch_bwd_wide_k<CELL, 8, 2>(v);
  if constexpr (CELL == kElman) {  // the other cells' chunks are wider than the registers hold
    if (ksplit == 4) return rows == 8 ? launch_bwd_wide_k<CELL, 4, 1>(v) : launch_bwd_wide_k<CELL, 4, 2>(v);
    if (ksplit == 2) return rows == 8 ? launch_bwd_wide_k<CELL, 2, 1>(v) : launch_bwd_wide_k<CELL, 2, 2>(v);
  }
  return kRegNoRoom;
}

}  // namespace frnn
