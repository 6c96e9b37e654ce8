// Reverse-time recurrence of narrow heads with R in the register file (see recurrent_reg.cuh).
//
// Groups, CTAs and the unit each thread owns are those of recurrent_reg_fwd.cu. Per step t a thread
//   1. adds up the partial dh_t of its unit and two batch rows (fixed order), the external gradient and the pointwise
//      carry, runs the cell backward and writes round_bf16(dg_t) to shared memory for ldmatrix (one CTA barrier),
//   2. multiplies with its warp's fragments of R_slice^T [D x GR*U] (rows = units p of h_{t-1}, k = gate rows of this CTA),
//   3. hands the accumulators to the owners of those units: two lanes swap halves so that each packet is 4 batch rows of
//      one unit, 16 bytes.
// The sums of step 2 run over the same gate rows in the same order as in the tcgen05 kernels, whose CTAs own 32 units (16
// where the width is not a multiple of 32), and step 1 adds them in the same order: every gradient is the same bits, whichever
// kernels a call takes.
//   LOCAL: D / 16 row tiles for D / 8 warps. 16 and 32 units: one sum per tile, which half of the warps run; 48 units: three
//          "sources" of 16 units each, two for the first half of the warps and one for the second.
//   else:  the sources are the CTAs of the cluster, packets travel by st.async. HALVES (odd multiples of 16): two sums per
//          tile, one for each 16 units of the CTA; the last CTA has units, and a sum, in its first half only.
// The state of step t - 1 stays in registers as the new state of the next iteration, and only the planes that the cell's
// derivative reads are fetched: an LSTM reads one history plane per step where reading both states at t and t - 1 takes four.
//
// Safe reuse: dg is double-buffered because a warp may still read dg_t when another has begun step t - 1; the partial
// sums of a parity are overwritten only after the CTA barrier of the step that read them; a TMA stage is refilled by the I/O
// warp after every warp has staged its outputs of the step that used it.
//
// Bound: the serial chain of a step. LSTM B8 N3 D256, 1513 cycles at 1845 MHz (see recurrent_reg_fwd.cu) = wait and reads 628 (the
// wait alone 173) + cell and barrier 137 + mma and scatter 612 + staging 127; 0.88 us per step of the call against 1.32 of the
// tcgen05 kernel; GRU B16 N24 D32 0.71 against 1.02; Elman B16 N12 D64 0.49 against 0.84; sLSTM B16 N4 D128 1.01 against 1.33.
#include "recurrent_reg.cuh"

namespace frnn {

namespace {

// History planes the cell's derivative reads: [first, first + count).
template <int CELL> struct HistPlanes;
template <> struct HistPlanes<kLSTM> { static constexpr int first = 1, count = 1; };
template <> struct HistPlanes<kSLSTM> { static constexpr int first = 1, count = 3; };
template <> struct HistPlanes<kGRU> { static constexpr int first = 0, count = 1; };
template <> struct HistPlanes<kElman> { static constexpr int first = 0, count = 1; };

template <int CELL, int KT, bool LOCAL, bool HALVES>
struct BwdRegCfg {
  using CT = CellTraits<CELL>;
  static constexpr int MTW = LOCAL ? 1 : (KT + 3) / 4;  // row tiles of a warp
  static constexpr int KTW = 2 * CT::GR;                // k tiles of a warp
  // Sums of a tile: one over all gate rows of the CTA; in a 48-unit CTA one for units 0 .. 15, 16 .. 31 and 32 .. 47 each, of
  // which a warp of the first half of the warps runs two; with HALVES one for each half of the CTA's units.
  static constexpr int CH = HALVES || (LOCAL && KT == 4) ? 2 : 1;
  static constexpr int MAX_SOURCES = LOCAL ? (KT == 4 ? 3 : 1) : 8 * CH;
  static constexpr int DG_BYTES = (CT::GR * (LOCAL ? KT * 16 : 32) * 16 + 511) / 512 * 512;  // two of them: the tiles stay 1 KB aligned
  static constexpr int GCL = CELL == kElman ? 0 : CT::GC;
  static constexpr int HP = HistPlanes<CELL>::first, HS = HistPlanes<CELL>::count;
  static constexpr int PLANE4 = kRegRows * kRegChunk * 4, PLANEC = kRegRows * kRegChunk * CT::CES;
  static constexpr int CHUNK = GCL * PLANEC + (HS + CT::S) * PLANE4;  // cache, state of step t - 1, external gradient
};

template <int CELL, int KT, bool LOCAL, bool HALVES>
__global__ void __launch_bounds__(reg_max_threads(KT, LOCAL), reg_min_blocks(CELL, KT, LOCAL, true))
frnn_bwd_reg_kernel(const BwdParams p, const float* history, const __grid_constant__ CUtensorMap cache_map,
                    const __grid_constant__ CUtensorMap hist_map, const __grid_constant__ CUtensorMap init_map,
                    const __grid_constant__ CUtensorMap dhist_map, const __grid_constant__ CUtensorMap dgr_map,
                    const __grid_constant__ CUtensorMap dwx_map, const int wx_bf16, const int own_dwx, const int stages_in_flight) {
  const int nst = LOCAL && KT > 2 ? stages_in_flight : kRegMaxStages;  // three only in a 48-unit CTA
  using Cfg = BwdRegCfg<CELL, KT, LOCAL, HALVES>;
  using CT = CellTraits<CELL>;
  constexpr int S = CT::S, MTW = Cfg::MTW, KTW = Cfg::KTW, CH = Cfg::CH, GCL = Cfg::GCL, HP = Cfg::HP, HS = Cfg::HS;

  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t s_part_bar[2];
  __shared__ __align__(8) uint64_t s_full[kRegMaxStages];
  __shared__ int s_gave_up;  // a compute warp of this CTA has stopped waiting (the flag in global memory is an L2 round trip away)
  __shared__ __align__(8) uint64_t s_out_full[kRegMaxSlots];  // outputs of a step staged by every warp

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane >> 2, c = lane & 3;
  const long long t_entry = clock64();
  const int D = p.D, N = p.N, T = p.T, B = p.B;
  const int nwarps = LOCAL ? (blockDim.x >> 5) - 1 : 4, U = nwarps * kRegUnitsPerWarp;
  const int C = LOCAL ? 1 : p.C;
  const int rank = LOCAL ? 0 : static_cast<int>(blockIdx.x % C), gid = blockIdx.x / C;
  const int n = gid % N, b0 = gid / N * kRegRows;
  const int sources = LOCAL ? Cfg::MAX_SOURCES : (HALVES ? D / 16 : C);
  const int part_bytes = sources * U * kRegRows * 4;  // one parity: [source][unit][8 batch rows] fp32
  const int chunks = (U + kRegChunk - 1) / kRegChunk, stage_bytes = chunks * Cfg::CHUNK;
  uint8_t* const dgbuf = smem;
  uint8_t* const part = smem + 2 * Cfg::DG_BYTES;
  uint8_t* const stages = part + 2 * part_bytes;
  uint8_t* const outs = stages + nst * stage_bytes;
  // Outputs of a step, staged per 32 units: dWx where it is a tensor of its own, and dg as the dR contraction wants it.
  const int slots = nst + 1;
  const int dwx_bytes = own_dwx ? CT::GW * (wx_bf16 ? kRegPlane<2> : kRegPlane<4>) : 0;
  const int out_chunk = reg_round_1k(dwx_bytes + CT::GR * kRegPlane<2>), out_slot = chunks * out_chunk;
  const volatile int* abort_flag = p.err;
  const uint64_t limit = p.wait_limit_ns;
  const int mute_from = p.err[4] != 0 ? p.err[5] : 0x7fffffff;            // test hook: nobody publishes from this iteration on
  const uint32_t jitter = wx_bf16 ? 0u : static_cast<uint32_t>(p.err[6]); // test hook (fp32 Wx): see jitter_stall
  const bool prof = p.err[3] != 0 && blockIdx.x == 0 && tid == 0;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&s_part_bar[i]), (LOCAL ? nwarps : 1) + 1);  // + the I/O warp: the tiles have landed
    for (int s = 0; s < nst; ++s) mbar_init(smem_u32(&s_full[s]), 1);
    for (int i = 0; i < slots; ++i) mbar_init(smem_u32(&s_out_full[i]), nwarps);
    s_gave_up = 0;
    fence_mbar_init();
  }
  for (int i = tid; i < 2 * Cfg::DG_BYTES / 16; i += blockDim.x)
    reinterpret_cast<uint4*>(dgbuf)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  // the packets carry all 8 columns whatever the number of batch rows in use
  const uint32_t part_tx = static_cast<uint32_t>(HALVES ? sources * min(U, D - rank * U) * kRegRows * 4 : part_bytes);
  if (tid == 0 && !LOCAL) {
    mbar_arrive_expect_tx(smem_u32(&s_part_bar[1]), part_tx);              // iteration 1 (the last one if T == 1)
    if (T >= 2) mbar_arrive_expect_tx(smem_u32(&s_part_bar[0]), part_tx);  // iteration 2
  }

  if (warp == nwarps) {
    // ---------------- I/O warp: tiles in, staged outputs out ----------------
    if (!LOCAL) cluster_sync_all();
    if (lane == 0) {
      auto fill = [&](int it, int s) {  // the operands of iteration `it`, step t
        const int t = T - 1 - it;
        const uint32_t bar = smem_u32(&s_full[s]);
        mbar_arrive_expect_tx(bar, static_cast<uint32_t>(stage_bytes));
        for (int i = 0; i < chunks; ++i) {
          uint32_t dst = smem_u32(stages + s * stage_bytes + i * Cfg::CHUNK);
          const int x = rank * U + i * kRegChunk;
          if (GCL > 0) tma_load_5d(dst, &cache_map, bar, x, n, b0, 0, t);
          dst += GCL * Cfg::PLANEC;
          if (t > 0) tma_load_5d(dst, &hist_map, bar, x, n, b0, HP, t - 1);
          else tma_load_5d(dst, &init_map, bar, x, n, b0, HP, 0);
          dst += HS * Cfg::PLANE4;
          tma_load_5d(dst, &dhist_map, bar, x, n, b0, 0, t);
        }
      };
      for (int it = 0; it < nst && it < T; ++it) fill(it, it);
      int stage = 0, slot = 0, next = 1;
      uint32_t phase = 0, next_phase = 0;
      // The barrier of the partial sums of iteration `it` also stands for its tiles: one wait per step on the compute
      // warps' chain, not two.
      auto announce = [&](int it) -> bool {
        if (it < T) {
          if (!mbar_wait_bounded<false, true>(smem_u32(&s_full[next]), next_phase & 1, limit, abort_flag)) {
            reg_report(p.err, kErrWaitWx, it);
            return false;
          }
          if (++next == nst) { next = 0; next_phase ^= 1u; }
        }
        mbar_arrive(smem_u32(&s_part_bar[it & 1]));
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
      for (int it = 1; it <= 2 && it <= T && ok; ++it) ok = announce(it);
      for (int it = 0; it < T && ok; ++it) {
        if (!staged(it)) {
          reg_report(p.err, kErrWaitEmpty, it);
          break;
        }
        // A warp that gave up on a wait sets the flag before it stages. Then the phase that the barrier is in may never
        // complete (another arrival would overrun its count), and a copy could be on its way into the stage: stop here.
        if (*reinterpret_cast<volatile int*>(&s_gave_up) != 0) break;
        // iteration it + 2 uses the barrier of iteration `it`, which every warp has left
        if (it >= 1 && it + 2 <= T) ok = announce(it + 2);
        for (int i = 0; i < chunks; ++i) {
          const uint32_t src = smem_u32(outs + slot * out_slot + i * out_chunk);
          const int x = rank * U + i * kRegChunk;
          if (own_dwx) tma_store_5d(&dwx_map, src, x, n, b0, 0, T - 1 - it);
          tma_store_5d(&dgr_map, src + dwx_bytes, x, n, b0, 0, T - 1 - it);
        }
        tma_store_commit();
        tma_store_wait_read<1>();  // the copies of the previous step have read their slot: see kRegMaxSlots
        if (it + nst < T) fill(it + nst, stage);
        if (++stage == nst) stage = 0;
        if (++slot == slots) { slot = 0; phase ^= 1u; }
      }
      tma_store_wait<0>();
    }
    __syncwarp();
  } else {
    // A fragments of R_slice^T: 8x8 blocks of R are loaded as they lie (gate rows x units p) and transposed in the warp.
    const int n_tiles = D / 16;
    const int part0 = LOCAL ? warp / n_tiles * CH : 0;   // first sum of this warp in the CTA ...
    const int source0 = LOCAL ? part0 : rank * CH;       // ... and in the group
    const int tile0 = LOCAL ? warp % n_tiles : warp;
    uint32_t a[MTW][KTW][4];
#pragma unroll
    for (int m = 0; m < MTW; ++m)
#pragma unroll
      for (int kt = 0; kt < KTW; ++kt)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          // block of 8 gate rows: tile kt of the gate-major rows; with two sums per warp, gate kt % GR of 16 units
          const int k8 = CH == 1 ? kt * 2 + (r >> 1) : kt % CT::GR * nwarps + 2 * (part0 + kt / CT::GR) + (r >> 1);
          const int g = k8 * 8 / U, u = k8 * 8 % U + q;
          const int pcol = (tile0 + (LOCAL ? 0 : 4 * m)) * 16 + 8 * (r & 1) + 2 * c;
          uint32_t v = 0u;
          if (g < CT::GR && pcol < D && source0 + (CH == 1 ? 0 : kt / CT::GR) < sources)
            v = __ldg(reinterpret_cast<const uint32_t*>(p.R + ((static_cast<size_t>(g) * N + n) * D + rank * U + u) * D + pcol));
          a[m][kt][r] = movmatrix_trans(v);
        }

    const int ul = warp * kRegUnitsPerWarp + q, d = rank * U + ul;
    const size_t ND = static_cast<size_t>(N) * D, BND = static_cast<size_t>(B) * ND;
    const size_t sBTND = static_cast<size_t>(T) * BND;
    const bool own = !HALVES || d < D;  // false in two warps of the last CTA, which take part in the products only
    bool act[2];
    float dcar[S][2], dbacc[CT::GB][2], sn[HS][2];
#pragma unroll
    for (int g = 0; g < CT::GB; ++g) dbacc[g][0] = dbacc[g][1] = 0.0f;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const size_t b = static_cast<size_t>(b0 + 2 * c + e);
      act[e] = own && b < static_cast<size_t>(B);
#pragma unroll
      for (int k = 0; k < S; ++k) dcar[k][e] = act[e] ? p.d_carry[k * BND + b * ND + static_cast<size_t>(n) * D + d] : 0.0f;
#pragma unroll
      for (int k = 0; k < HS; ++k)
        sn[k][e] = act[e] ? history[(HP + k) * sBTND + ((b * T + T - 1) * N + n) * D + d] : 0.0f;
    }
    const int uc = (warp & 3) * kRegUnitsPerWarp + q;  // unit inside the staged 32
    const uint32_t off_q = reg_tile_offset<2>(q, (warp & 3) * kRegUnitsPerWarp + 2 * c);
    uint8_t* const my_chunk = stages + (warp >> 2) * Cfg::CHUNK;
    uint8_t* const my_out = outs + (warp >> 2) * out_chunk;
    uint8_t* out = my_out;
    const int compute_threads = nwarps * 32;
    const bool v1 = p.slstm_v1 != 0, zero_first = p.slstm_zero_first != 0, cut = p.cut_recurrent != 0, clip_on = p.grad_clip > 0.0f;
    const float grad_clip = p.grad_clip;
    // where this lane's packets of a tile go: the row q or q + 8 of the tile, four batch rows
    const uint32_t row_off = static_cast<uint32_t>((q + 8 * (c & 1)) * (kRegRows * 4) + (c >> 1) * 16);
    uint32_t dst_part[MTW], dst_bar[MTW];
#pragma unroll
    for (int m = 0; m < MTW; ++m) {
      const int tile = tile0 + (LOCAL ? 0 : 4 * m);
      if (LOCAL) {
        dst_part[m] = smem_u32(part) + (source0 * U + tile * 16) * (kRegRows * 4) + row_off;
        dst_bar[m] = 0u;
      } else {
        const int owner = tile < n_tiles ? tile / 2 : rank;  // 32 units, two tiles
        dst_part[m] = map_to_cta(smem_u32(part) + (source0 * U + (tile & 1) * 16) * (kRegRows * 4) + row_off, owner);
        dst_bar[m] = map_to_cta(smem_u32(&s_part_bar[0]), owner);
      }
    }

    bool dead = false;  // warp-uniform: after a failed wait the warp walks on without waiting
    auto give_up = [&](int code, int it) {
      if (lane == 0) reg_report(p.err, code, it);
      dead = true;
      *reinterpret_cast<volatile int*>(&s_gave_up) = 1;
    };
    float cache[CT::GC][2], sp[HS][2], dh[S][2];
    int in_stage = 0, slot = 0;
    auto read_stage = [&]() {
      const uint8_t* sb = my_chunk + in_stage * stage_bytes;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int row = 2 * c + e;
#pragma unroll
        for (int g = 0; g < GCL; ++g) cache[g][e] = ld_cache<CT::CES>(sb + g * Cfg::PLANEC + reg_tile_offset<CT::CES>(row, uc), 0);
        const uint8_t* f = sb + GCL * Cfg::PLANEC + reg_tile_offset<4>(row, uc);
#pragma unroll
        for (int k = 0; k < HS; ++k) sp[k][e] = *reinterpret_cast<const float*>(f + k * Cfg::PLANE4);
        f += HS * Cfg::PLANE4;
#pragma unroll
        for (int k = 0; k < S; ++k) dh[k][e] = *reinterpret_cast<const float*>(f + k * Cfg::PLANE4);
      }
      if (++in_stage == nst) in_stage = 0;
    };
    if (!LOCAL) cluster_sync_all();
    if (prof) p.err[20] = static_cast<int>(clock64() - t_entry);

    if (!mbar_wait_warp<false>(smem_u32(&s_full[0]), 0, limit, abort_flag)) give_up(kErrWaitWx, 0);
    constexpr int kSrc = HALVES ? 8 : Cfg::MAX_SOURCES;  // sources read at once
    long long pc[6] = {0, 0, 0, 0, 0, 0};
    for (int it = 0; it <= T; ++it) {
      if (jitter != 0u) { jitter_stall(jitter, static_cast<uint32_t>(warp), static_cast<uint32_t>(it)); __syncwarp(); }
      const int t = T - 1 - it;
      float ds[S][2];
      float2 v[kSrc];
#pragma unroll
      for (int k = 0; k < kSrc; ++k) v[k] = make_float2(0.0f, 0.0f);
      const long long c1 = prof ? clock64() : 0;
      long long cw = c1;
      if (it >= 1) {
        const int pb = it & 1;
        if (!dead && !mbar_wait_warp<!LOCAL>(smem_u32(&s_part_bar[pb]), ((it - 1) >> 1) & 1, limit, abort_flag)) give_up(kErrWaitPart, it);
        cw = prof ? clock64() : 0;
        if (!cut) {
          const uint8_t* pbuf = part + pb * part_bytes + ul * (kRegRows * 4) + c * 8;
#pragma unroll
          for (int k = 0; k < kSrc; ++k)
            if (k < sources) v[k] = *reinterpret_cast<const float2*>(pbuf + k * U * (kRegRows * 4));
        }
      }
      if (it < T) read_stage();
#pragma unroll
      for (int k = 0; k < S; ++k)
#pragma unroll
        for (int e = 0; e < 2; ++e) ds[k][e] = it < T ? dcar[k][e] + dh[k][e] : dcar[k][e];
#pragma unroll
      for (int k = 0; k < kSrc; ++k) { ds[0][0] += v[k].x; ds[0][1] += v[k].y; }
      if (HALVES && it >= 1 && !cut) {
        const uint8_t* pbuf = part + (it & 1) * part_bytes + ul * (kRegRows * 4) + c * 8;
#pragma unroll
        for (int k = 0; k < kSrc; ++k)
          v[k] = kSrc + k < sources ? *reinterpret_cast<const float2*>(pbuf + (kSrc + k) * U * (kRegRows * 4)) : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int k = 0; k < kSrc; ++k) { ds[0][0] += v[k].x; ds[0][1] += v[k].y; }
      }
      if (clip_on && it >= 1 && it < T) {
        // the gradient carried into h_t from step t + 1 (total minus the external part) is complete here: clip it
#pragma unroll
        for (int e = 0; e < 2; ++e) ds[0][e] = clip_sym(ds[0][e] - dh[0][e], grad_clip) + dh[0][e];
      }
      const long long c2 = prof ? clock64() : 0;
      if (it == T) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (act[e]) {
#pragma unroll
            for (int k = 0; k < S; ++k)
              p.d_initial[k * BND + static_cast<size_t>(b0 + 2 * c + e) * ND + static_cast<size_t>(n) * D + d] = ds[k][e];
          }
        break;
      }
      float dgr[CT::GR][2], dgw[CT::GW][2];
      const bool take_i = CELL == kSLSTM && t == 0 && zero_first;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float cj[CT::GC], snj[S], spj[S], dsj[S], gr[CT::GR], gw[CT::GW], gb[CT::GB];
#pragma unroll
        for (int g = 0; g < GCL; ++g) cj[g] = cache[g][e];
#pragma unroll
        for (int k = 0; k < S; ++k) {
          snj[k] = k >= HP && k < HP + HS ? sn[k >= HP ? k - HP : 0][e] : 0.0f;
          spj[k] = k >= HP && k < HP + HS ? sp[k >= HP ? k - HP : 0][e] : 0.0f;
          dsj[k] = ds[k][e];
        }
        cell_backward<CELL>(cj, spj, snj, dsj, gr, gw, gb, take_i, v1);
        // rows past the batch hold zeros where the cell divides: their gradients are dropped
#pragma unroll
        for (int k = 0; k < S; ++k) dcar[k][e] = act[e] ? dsj[k] : 0.0f;
#pragma unroll
        for (int g = 0; g < CT::GR; ++g) dgr[g][e] = act[e] ? gr[g] : 0.0f;
#pragma unroll
        for (int g = 0; g < CT::GW; ++g) dgw[g][e] = act[e] ? gw[g] : 0.0f;
      }
      uint32_t dgp[CT::GR];
      const uint32_t dgs = smem_u32(dgbuf) + (it & 1) * Cfg::DG_BYTES;
#pragma unroll
      for (int g = 0; g < CT::GR; ++g) {
        dgp[g] = pack_bf16x2(dgr[g][0], dgr[g][1]);
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(dgs + (g * nwarps + warp) * 128 + lane * 4), "r"(dgp[g]) : "memory");
      }
#pragma unroll
      for (int k = 0; k < HS; ++k) { sn[k][0] = sp[k][0]; sn[k][1] = sp[k][1]; }
      asm volatile("bar.sync 1, %0;" ::"r"(compute_threads) : "memory");
      const long long c3 = prof ? clock64() : 0;
      const int nb = (it + 1) & 1;
      const bool publish = !dead && it < mute_from;
      if (!LOCAL || source0 < sources) {
        float acc[CH][MTW][4];
#pragma unroll
        for (int h = 0; h < CH; ++h)
#pragma unroll
          for (int m = 0; m < MTW; ++m)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[h][m][r] = 0.0f;
        if constexpr (CH == 1) {
#pragma unroll
          for (int k2 = 0; k2 < KTW / 2; ++k2) {
            uint32_t bf[4];
            ldsm_x4_trans(dgs + lane * 16 + k2 * 512, bf);
#pragma unroll
            for (int m = 0; m < MTW; ++m) mma_bf16_16816(acc[0][m], a[m][2 * k2], bf[0], bf[1]);
#pragma unroll
            for (int m = 0; m < MTW; ++m) mma_bf16_16816(acc[0][m], a[m][2 * k2 + 1], bf[2], bf[3]);
          }
        } else {
          // gate g: the blocks of four warps, two for each sum; a sum past the last source is computed and dropped
#pragma unroll
          for (int g = 0; g < CT::GR; ++g) {
            uint32_t bf[4];
            ldsm_x4_trans(dgs + (g * nwarps + 2 * part0) * 128 + lane * 16, bf);
#pragma unroll
            for (int m = 0; m < MTW; ++m) mma_bf16_16816(acc[0][m], a[m][g], bf[0], bf[1]);
#pragma unroll
            for (int m = 0; m < MTW; ++m) mma_bf16_16816(acc[CH - 1][m], a[m][CT::GR + g], bf[2], bf[3]);
          }
        }
#pragma unroll
        for (int h = 0; h < CH; ++h)
#pragma unroll
          for (int m = 0; m < MTW; ++m) {
            const float(&v)[4] = acc[h][m];
            // rows q / q + 8, columns 2c, 2c + 1 -> even lanes: row q, columns 2c .. 2c + 3; odd lanes: row q + 8, 2c - 2 .. 2c + 1
            const float x0 = __shfl_xor_sync(0xffffffffu, (c & 1) ? v[0] : v[2], 1);
            const float x1 = __shfl_xor_sync(0xffffffffu, (c & 1) ? v[1] : v[3], 1);
            const float4 w = (c & 1) ? make_float4(x0, x1, v[2], v[3]) : make_float4(v[0], v[1], x0, x1);
            if constexpr (LOCAL) {
              if (publish && source0 + h < sources)
                asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst_part[m] + nb * part_bytes + h * U * (kRegRows * 4)),
                             "f"(w.x), "f"(w.y), "f"(w.z), "f"(w.w) : "memory");
            } else {
              if (publish && tile0 + 4 * m < n_tiles && (!HALVES || source0 + h < sources))
                st_async_v4_b32(dst_part[m] + nb * part_bytes + h * U * (kRegRows * 4), __float_as_uint(w.x), __float_as_uint(w.y), __float_as_uint(w.z),
                                __float_as_uint(w.w), dst_bar[m] + nb * 8);
            }
          }
      }
      if constexpr (LOCAL) {
        __syncwarp();
        if (lane == 0 && publish) mbar_arrive(smem_u32(&s_part_bar[nb]));
      }
      // this parity's partial sums were complete at the wait above: armed for iteration it + 2
      if (!LOCAL && tid == 0 && !dead && it >= 1 && it + 2 <= T) mbar_arrive_expect_tx(smem_u32(&s_part_bar[it & 1]), part_tx);
      const long long c4 = prof ? clock64() : 0;
      // outputs, while the partial sums of the next step are on their way
#pragma unroll
      for (int g = 0; g < CT::GR; ++g) reg_stage_16(out + dwx_bytes + g * kRegPlane<2>, off_q, dgp[g]);
      if (own_dwx) {
#pragma unroll
        for (int g = 0; g < CT::GW; ++g) {
          if (wx_bf16) reg_stage_16(out + g * kRegPlane<2>, off_q, pack_bf16x2(dgw[g][0], dgw[g][1]));
          else reg_stage_f32(out + g * kRegPlane<4>, c, uc, dgw[g][0], dgw[g][1]);
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_out_full[slot]));
#pragma unroll
      for (int g = 0; g < CT::GB; ++g)
#pragma unroll
        for (int e = 0; e < 2; ++e) dbacc[g][e] += CELL != kGRU ? dgw[g][e] : (g == 0 ? dgr[0][e] : dgw[g > 0 ? g - 1 : 0][e]);  // as cell_backward's gb
      out += out_slot;
      if (++slot == slots) { slot = 0; out = my_out; }
      const long long c5 = prof ? clock64() : 0;
      if (prof) {
        pc[0] += clock64() - c1; pc[1] += c2 - c1; pc[2] += c3 - c2; pc[3] += c5 - c4; pc[4] += c4 - c3; pc[5] += cw - c1;
      }
    }
    if (prof) {  // the slots of the tcgen05 kernels' phase timers that have a counterpart here
      p.err[15] = static_cast<int>(pc[0]);  // the whole step
      p.err[9] = static_cast<int>(pc[1]);   // wait for the partial sums and tiles, their sum
      p.err[10] = static_cast<int>(pc[2]);  // cell, dg to shared memory, CTA barrier
      p.err[11] = static_cast<int>(pc[3]);  // outputs staged
      p.err[12] = static_cast<int>(pc[4]);  // mma and scatter
      p.err[13] = static_cast<int>(pc[5]);  // wait alone
    }
    // bias gradient of the 8 batch rows, added in their order
#pragma unroll
    for (int g = 0; g < CT::GB; ++g) {
      float v = 0.0f;
#pragma unroll
      for (int k = 0; k < kRegRows; ++k) v += __shfl_sync(0xffffffffu, dbacc[g][k & 1], (lane & ~3) + (k >> 1));
      if (c == 0 && own) {
        float* dst = p.db_part + ((static_cast<size_t>(b0 / p.db_rows) * CT::GB + g) * N + n) * D + d;
        // an entry of 16 rows gets at most two addends on top of the launcher's zeros: the order cannot matter, but the sum may
        // differ in its last bits from the 16 rows added one by one
        if (p.db_rows == kRegRows) *dst = v;
        else atomicAdd(dst, v);
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

template <int CELL, int KT, bool LOCAL, bool HALVES = false>
int launch_bwd_reg(const BwdParams& p, const void* cache, const float* history, const float* initial,
                   const float* d_history, int wx_bf16, cudaStream_t stream, bool ask) {
  using Cfg = BwdRegCfg<CELL, KT, LOCAL, HALVES>;
  using CT = CellTraits<CELL>;
  const int U = LOCAL ? p.D : kRegClusterUnits, C = (p.D + U - 1) / U;
  const int stage = reg_chunks(U) * Cfg::CHUNK;
  // cells whose W-gates are their R-gates may have one bf16 buffer for dWx and dg
  const bool own_dwx = !wx_bf16 || CELL == kGRU || p.dwx != static_cast<void*>(p.dgr);
  const int out_slot = reg_chunks(U) * reg_round_1k(kRegRows * kRegChunk * (CT::GR * 2 + (own_dwx ? CT::GW * (wx_bf16 ? 2 : 4) : 0)));
  // prefetch depth: 4 steps, 3 where only that lets two CTAs share an SM
  const auto bytes = [&](int st) {
    return 2 * Cfg::DG_BYTES + 2 * (LOCAL ? Cfg::MAX_SOURCES : (HALVES ? p.D / 16 : C)) * U * kRegRows * 4 + st * stage + (st + 1) * out_slot;
  };
  const int nst = LOCAL && KT > 2 ? reg_stages(bytes(kRegMaxStages), bytes(kRegMaxStages - 1)) : kRegMaxStages;
  const int smem = bytes(nst);
  if (smem > kRegSmemLimit) return -2;
  const int D = p.D, N = p.N, B = p.B;
  const uint64_t nd = static_cast<uint64_t>(N) * D, uT = p.T, uB = p.B;
  // bulk stores start on 16-byte boundaries; the tcgen05 kernels write these outputs with plain stores
  if (((reinterpret_cast<uintptr_t>(p.dwx) | reinterpret_cast<uintptr_t>(p.dgr)) & 15u) != 0) return kRegNoRoom;
  auto kern = frnn_bwd_reg_kernel<CELL, KT, LOCAL, HALVES>;
  BwdParams q = p;
  q.C = C;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(p.N * reg_batch_tiles(p.B) * C));
  cfg.blockDim = dim3(static_cast<unsigned>(U / kRegUnitsPerWarp * 32 + 32));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(C);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = LOCAL ? 0 : 1;
  // whether the call is taken at all comes first: one that is not pays for nothing else
  const int rc = reg_room(reinterpret_cast<const void*>(kern), cfg, C, p.N, p.B, p.D);
  if (rc != 0 || ask) return rc != 0 ? rc : kRegTaken;
  CUtensorMap cache_map, hist_map, init_map, dhist_map, dgr_map, dwx_map;
  if (reg_tile_map(&hist_map, history, 4, D, N, B, CT::S, p.T, uT * nd, uB * uT * nd, nd, Cfg::HS) != 0 ||
      reg_tile_map(&dhist_map, d_history, 4, D, N, B, CT::S, p.T, uT * nd, uB * uT * nd, nd, CT::S) != 0 ||
      reg_tile_map(&init_map, initial, 4, D, N, B, CT::S, 1, nd, uB * nd, nd, Cfg::HS) != 0 ||
      reg_tile_map(&dgr_map, p.dgr, 2, D, N, B, CT::GR, p.T, uT * CT::GR * nd, nd, CT::GR * nd, CT::GR) != 0)
    return -4;
  cache_map = hist_map;  // Elman has no cache: a valid map that is never used
  if (Cfg::GCL > 0 &&
      reg_tile_map(&cache_map, cache, CT::CES, D, N, B, CT::GC, p.T, uT * CT::GC * nd, nd, CT::GC * nd, CT::GC) != 0)
    return -4;
  dwx_map = dgr_map;
  if (own_dwx &&
      reg_tile_map(&dwx_map, p.dwx, wx_bf16 ? 2 : 4, D, N, B, CT::GW, p.T, uT * CT::GW * nd, nd, CT::GW * nd, CT::GW) != 0)
    return -4;
  if (p.db_rows != kRegRows) {
    const size_t tiles = static_cast<size_t>((p.B + p.db_rows - 1) / p.db_rows);
    const cudaError_t e = cudaMemsetAsync(p.db_part, 0, tiles * CT::GB * p.N * p.D * sizeof(float), stream);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, q, history, cache_map, hist_map, init_map, dhist_map, dgr_map, dwx_map,
                                             wx_bf16, own_dwx ? 1 : 0, nst));
}

template <int CELL, int KT>
int launch_bwd_reg_cluster(const BwdParams& p, const void* cache, const float* history, const float* initial,
                           const float* d_history, int wx_bf16, cudaStream_t s, bool ask) {
  if (p.D % kRegClusterUnits != 0) {
    // The odd multiples of 16 begin at 80. The sLSTM at 208 and 240 units needs all 255 registers and is no faster here than
    // on the tcgen05 kernel: T128 N1, forward and backward, 399 us against 378 at B4 D208 and 488 against 478 at B48 D240.
    if constexpr (KT > 4 && !(CELL == kSLSTM && KT > 12))
      return launch_bwd_reg<CELL, KT, false, true>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    else
      return kRegNoRoom;
  }
  return launch_bwd_reg<CELL, KT, false>(p, cache, history, initial, d_history, wx_bf16, s, ask);
}

template <int CELL>
int launch_bwd_reg_cell(const BwdParams& p, const void* cache, const float* history, const float* initial,
                        const float* d_history, int wx_bf16, cudaStream_t s, bool ask) {
  switch (reg_k_tiles(p.D)) {
    case 2: return launch_bwd_reg<CELL, 2, true>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    case 4:
      return reg_local(p.D) ? launch_bwd_reg<CELL, 4, true>(p, cache, history, initial, d_history, wx_bf16, s, ask)
                            : launch_bwd_reg_cluster<CELL, 4>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    case 6: return launch_bwd_reg_cluster<CELL, 6>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    case 8: return launch_bwd_reg_cluster<CELL, 8>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    case 10: return launch_bwd_reg_cluster<CELL, 10>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    case 12: return launch_bwd_reg_cluster<CELL, 12>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    case 14: return launch_bwd_reg_cluster<CELL, 14>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    case 16: return launch_bwd_reg_cluster<CELL, 16>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    default: return -2;
  }
}

}  // namespace

int backward_reg_dispatch(int cell, const BwdParams& p, const void* cache, const float* history, const float* initial,
                          const float* d_history, int wx_bf16, cudaStream_t s, bool ask) {
  switch (cell) {
    case kLSTM: return launch_bwd_reg_cell<kLSTM>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    case kSLSTM: return launch_bwd_reg_cell<kSLSTM>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    case kGRU: return launch_bwd_reg_cell<kGRU>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    case kElman: return launch_bwd_reg_cell<kElman>(p, cache, history, initial, d_history, wx_bf16, s, ask);
    default: return -1;
  }
}

}  // namespace frnn
