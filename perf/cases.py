"""Workloads whose speed this repository watches: what its users run through the public entry points.

Every case is one pass of a recurrent layer: a decoding step or a streamed piece of a sequence (forward only, small), a
whole sequence without gradients, or a training pass (forward, then the gradients of every input). Shapes come from the
benchmark configurations, the published head-width sweep (heads x width = 768) and the tests. ``draw`` gives further
cases of the same ranges.
"""

from __future__ import annotations

import math

import torch

from flashrnn_b200 import PreparedSequence, flashrnn, flashrnn_projected, flashrnn_torch

# cell -> (recurrent gates, Wx gates, bias gates, states)
CELLS = {"lstm": (4, 4, 4, 2), "slstm": (4, 4, 4, 4), "gru": (3, 3, 4, 1), "elman": (1, 1, 1, 1)}

# A case:
#   kind   "decode"    a few steps without gradients through flashrnn(), bf16 weights, the carry of the previous call
#          "stream"    a captured PreparedSequence that writes the hidden states of a piece of a sequence
#          "infer"     a whole sequence without gradients; "inputs" > 0: with the input projection in front
#          "train"     forward and the gradients of Wx (or x and W), R, b and the initial state
#   cell, B, T, N, D, dtype ("bfloat16" or "float32": the type of Wx)
#   states True: the call starts from a given state (and hands its gradient back), False: from zeros
#   carry  True: the loss also depends on the last state (truncated back-propagation over pieces)


def _case(name, kind, cell, B, T, N, D, dtype="bfloat16", states=True, carry=False, inputs=0):
    out = {"kind": kind, "cell": cell, "B": B, "T": T, "N": N, "D": D, "dtype": dtype, "states": states, "carry": carry,
           "inputs": inputs}
    if name:
        out["name"] = name
    return out


def listed():
    return [
        # serving: one token for four streams, the call that a decoding loop makes
        _case("decode_lstm_B4_T1_N3_D256", "decode", "lstm", 4, 1, 3, 256),
        # serving: a short piece of a stream on fixed buffers, replayed as a graph; one wide head
        _case("stream_lstm_B4_T16_N1_D768", "stream", "lstm", 4, 16, 1, 768),
        # the small training shape of the tests, fp32 inputs
        _case("train_lstm_fp32_B8_T256_N1_D64", "train", "lstm", 8, 256, 1, 64, "float32"),
        # the headline training step
        _case("train_lstm_B8_T1024_N3_D256", "train", "lstm", 8, 1024, 3, 256),
        # sLSTM over long sequences, from the zero state
        _case("train_slstm_B16_T2048_N4_D128", "train", "slstm", 16, 2048, 4, 128, states=False),
        # head-width sweep: many narrow heads, the gated and the ungated cell
        _case("train_gru_B16_T1024_N24_D32", "train", "gru", 16, 1024, 24, 32),
        _case("train_elman_B16_T1024_N12_D64", "train", "elman", 16, 1024, 12, 64),
        # head-width sweep: one wide head
        _case("train_lstm_B16_T1024_N1_D768", "train", "lstm", 16, 1024, 1, 768),
        # ragged everywhere: odd batch and length, a width that no kernel tiles, fp32, gradient through the carry
        _case("train_gru_fp32_B13_T333_N2_D200", "train", "gru", 13, 333, 2, 200, "float32", carry=True),
        # a layer's forward pass over a batch of sequences, with its input projection
        _case("infer_lstm_proj_B64_T512_N2_D384", "infer", "lstm", 64, 512, 2, 384, inputs=768),
        # a head wider than one GPU's on-chip weights allow without splitting
        _case("train_lstm_B16_T128_N1_D2048", "train", "lstm", 16, 128, 1, 2048),
        # the largest batch: one GPU's share of a 32-head layer
        _case("train_lstm_B256_T2048_N4_D128", "train", "lstm", 256, 2048, 4, 128, states=False),
    ]


_ITEMS_MAX = 256 * 2048 * 4 * 128          # (batch, step, unit) triples of the largest listed case
_MACS_MAX = _ITEMS_MAX * 4 * 128           # its multiply-adds of one contraction with R


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("decode", "stream", "infer", "infer", "train", "train", "train", "train"))
    cell = rng.choice(("lstm", "lstm", "slstm", "gru", "elman"))
    dtype = rng.choice(("bfloat16", "bfloat16", "float32"))
    D = rng.choice((16, 32, 48, 64, 96, 128, 160, 192, 256, 320, 384, 512, 640, 768) + tuple(_log_int(rng, 16, 768) for _ in range(5)))
    N = max(1, min(48, _log_int(rng, 256, 1536) // D))
    inputs = 0
    if kind in ("decode", "stream"):
        B = _log_int(rng, 1, 64)
        T = _log_int(rng, 1, 4) if kind == "decode" else _log_int(rng, 4, 64)
        if kind == "stream":
            m = 16 if D <= 512 else 64    # prepared sequences take widths that the kernels tile and what one launch holds
            D = (D + m - 1) // m * m
            B = min(B, 16) if D > 512 else B
    else:
        B = _log_int(rng, 1, 96)
        T = _log_int(rng, 64, 1536)
        if kind == "infer" and rng.random() < 0.5:
            inputs = 8 * _log_int(rng, 16, 128)
            D, N = (D + 15) // 16 * 16, max(1, N)
            while CELLS[cell][1] * N * D % 64:
                N += 1
    macs = B * T * N * D * D * CELLS[cell][0]
    if macs > _MACS_MAX // 4 or B * T * N * D > _ITEMS_MAX // 4:
        B = max(1, int(B * min(_MACS_MAX / 4 / macs, _ITEMS_MAX / 4 / (B * T * N * D))))
    states = kind in ("decode", "stream") or rng.random() < 0.6
    return _case(None, kind, cell, B, T, N, D, dtype, states, kind == "train" and states and rng.random() < 0.3, inputs)


def prepare(case, seed):
    cell, B, T, N, D = (case[k] for k in ("cell", "B", "T", "N", "D"))
    gr, gw, gb, S = CELLS[cell]
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    wx_dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32

    def randn(*shape, dtype=torch.float32, scale=1.0):
        return (torch.randn(shape, generator=g, device=dev, dtype=torch.float32) * scale).to(dtype)

    R = randn(gr, N, D, D, scale=D ** -0.5)
    b = randn(gb, N, D, scale=0.1)
    if cell == "slstm":                       # the usual forget-gate bias
        b[1] = torch.rand((N, D), generator=g, device=dev) * 3.0 + 3.0
    states = None
    if case["states"]:
        states = randn(S, B, 1, N, D, scale=0.5)
        if cell == "slstm":
            states[2] = states[2].abs() + 1.0  # a normaliser carried over from earlier steps is at least one
    st = {"case": dict(case)}
    if case["inputs"]:
        st["x"] = randn(B, T, case["inputs"], dtype=torch.bfloat16)
        st["W"] = randn(gw * N * D, case["inputs"], dtype=torch.bfloat16, scale=case["inputs"] ** -0.5)
    else:
        st["wx"] = randn(B, T, gw, N, D, dtype=wx_dtype)
    if case["kind"] in ("decode", "stream") or case["inputs"]:
        R = R.to(torch.bfloat16)               # a serving program holds rounded weights
    st.update(R=R, b=b, states=states)
    if case["kind"] == "stream":
        st["seq"] = PreparedSequence(st["wx"], R, b, states, cell, output_mode="hidden").capture()
    if case["kind"] == "train":
        st["leaves"] = [t.requires_grad_(True) for t in (st["wx"], R, b, states) if t is not None]
        st["dh"] = randn(B, T, N, D)
        if case["carry"]:
            st["dc"] = randn(S, B, 1, N, D)
    return st


def run(state):
    case = state["case"]
    cell, kind, dtype = case["cell"], case["kind"], case["dtype"]
    if kind == "stream":
        return state["seq"].run()
    if kind != "train":
        with torch.no_grad():
            if case["inputs"]:
                return flashrnn_projected(state["x"], state["W"], state["R"], state["b"], state["states"], function=cell,
                                          dtype=dtype)
            return flashrnn(state["wx"], state["R"], state["b"], state["states"], function=cell, dtype=dtype)
    if dtype == "float32" and state["states"] is not None:
        hist, carry = flashrnn_torch(state["wx"], state["R"], state["b"], state["states"], cell=cell,
                                     numerics="fp32_state_bf16_mma")
    else:
        hist, carry = flashrnn(state["wx"], state["R"], state["b"], state["states"], function=cell, dtype=dtype)
    # the next layer consumes the hidden states and hands their gradient back
    outs, grads = [hist[0]], [state["dh"]]
    if case["carry"]:
        outs.append(carry)
        grads.append(state["dc"])
    return (hist.detach(), carry.detach()) + torch.autograd.grad(outs, state["leaves"], grads)


def work(case):
    cell, B, T, N, D = (case[k] for k in ("cell", "B", "T", "N", "D"))
    gr, gw, gb, S = CELLS[cell]
    es = 2 if case["dtype"] == "bfloat16" else 4
    items = B * T * N * D
    r_bytes = gr * N * D * D * (2 if case["kind"] in ("decode", "stream") or case["inputs"] else 4)
    small = gb * N * D * 4 + (2 if case["states"] else 1) * S * B * N * D * 4     # biases, first and last states
    flops = 2.0 * gr * D * items                                                   # R h
    total = r_bytes + small
    if case["inputs"]:
        total += (B * T + gw * N * D) * case["inputs"] * 2
        flops += 2.0 * B * T * case["inputs"] * gw * N * D
    else:
        total += items * gw * es
    total += items * 4 * (1 if case["kind"] == "stream" else S)                    # hidden states / all states
    if case["kind"] == "train":
        # gradients: dh in, dWx out, dR, db and the initial state's out; two more contractions with R / for dR
        total += items * 4 + items * gw * es + r_bytes + small
        flops *= 3.0
    return {"bytes": float(total), "flops": flops}


def tolerance(case):
    # R and the recurrent operands (h forward, gate gradients backward) are bf16 in every case, states and sums fp32
    return {"rel": 1e-2}
