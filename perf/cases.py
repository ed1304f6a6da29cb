"""The work that users of this package have it do, as cases that can be timed and compared.

A case is one pass through the public entry points (`window_matmul`, `window_softmax`, `unwindow_matmul`):

  mode "chain"      window_matmul -> unwindow_matmul and the backward of both: the two operators as they stand
  mode "attention"  window_matmul -> window_softmax -> unwindow_matmul and its backward: a training step of windowed attention
  mode "forward"    the attention block without gradients: inference

over (batch, heads, rows, hidden) tensors with window `window`, in one of the operand layouts that callers have:

  layout "heads"  q, k, v contiguous (batch, heads, rows, hidden), the key passed as its transposed view
  layout "bnm"    the key stored the way the operator takes it, contiguous (batch, heads, hidden, rows)
  layout "proj"   q, k, v are the (batch, heads, rows, hidden) views of (batch, rows, heads * hidden) projections

`autocast` runs a float32 case under torch.autocast("cuda"), where the two operators compute in float16.
"""
import contextlib
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("pytorch-window-matmul_b200"))   # (the working folder is the root of the repository)
from window_matmul import unwindow_matmul, window_matmul, window_softmax  # noqa: E402

_DTYPES = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}


def _case(name, mode, dtype, batch, heads, rows, hidden, window, layout="heads", autocast=False):
    case = dict(mode=mode, dtype=dtype, batch=batch, heads=heads, rows=rows, hidden=hidden, window=window, layout=layout, autocast=autocast)
    return dict(case, name=name) if name else case


def listed():
    return [
        # The headline of the benchmark: the attention band of an 8 x 12-head base model with window 2 x 256, in 16 bits ...
        _case("band_train_bf16", "chain", "bfloat16", 8, 12, 4096, 64, 256),
        # ... and the same job in float32, where the results keep the exact order of summation.
        _case("band_train_fp32", "chain", "float32", 8, 12, 4096, 64, 256),
        # A small float32 step (benchmark configuration 1): few tiles, the launches and the host count.
        _case("small_train_fp32", "chain", "float32", 4, 1, 1024, 64, 64),
        # Narrow windows over many short sequences (configuration 3): all memory traffic.
        _case("narrow_train_fp16", "chain", "float16", 1024, 1, 2048, 32, 8),
        # One long sequence with a wide window and a large head (configuration 4): the largest case.
        _case("long_train_bf16", "chain", "bfloat16", 1, 16, 65536, 128, 512),
        # A full attention block, forward and backward (configuration 5).
        _case("attention_train_bf16", "attention", "bfloat16", 4, 16, 16384, 64, 384),
        # The size of the reference's own tests (2 x 1 x 32 x 3, window 4): what one call costs at the least.
        _case("tiny_train_fp32", "chain", "float32", 2, 1, 32, 3, 4),
        # Inference on one short input.
        _case("short_forward_bf16", "forward", "bfloat16", 1, 12, 512, 64, 64),
        # Inference on one document, whose length is whatever it is.
        _case("document_forward_fp16", "forward", "float16", 1, 12, 3001, 64, 128),
        # Training with sizes that fit no tile: odd length, a head size of 80, a window that is no power of two.
        _case("ragged_train_bf16", "attention", "bfloat16", 4, 12, 1111, 80, 75),
        # Mixed-precision training as a module does it: float32 projections viewed per head, autocast.
        _case("projection_train_amp", "attention", "float32", 4, 12, 2048, 64, 256, "proj", True),
        # The key stored as (hidden, rows), the layout of the reference's usage example.
        _case("key_bnm_train_fp16", "chain", "float16", 2, 16, 4096, 128, 128, "bnm"),
    ]


#: No drawn case asks for more operations or moves more bytes than configuration 2 does (the longest listed pass, in float32).
_MOST_FLOPS, _MOST_BYTES = 1.5e11, 2.5e9


def _log_between(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    mode = rng.choice(["chain", "attention", "forward"])
    dtype, autocast = rng.choice([("bfloat16", False), ("float16", False), ("float32", False), ("float32", True)])
    layout = rng.choice(["heads", "heads", "bnm", "proj"])
    # head sizes: the usual ones, now and then any
    hidden = rng.choice([32, 64, 64, 64, 128, 128, 16, 48, 80, 96, rng.randint(3, 128)])
    # windows: an attention block has one of the usual sizes, as often as not with a few positions more; the bare
    # operators meet any.  Lengths: as often a round number as not
    if mode == "chain":
        window = _log_between(rng, 2, 512)
        if window >= 16 and rng.random() < 0.5:
            window = window // 16 * 16
    else:
        window = rng.choice([rng.randint(2, 16), 16, 32, 64, 64, 128, 128, 192, 256, 256, 384, 512])
        if window >= 16 and rng.random() < 0.5:
            window += rng.randint(1, 15)
    rows = _log_between(rng, 32, 65536)
    if rng.random() < 0.5:
        rows = max(32, rows // 32 * 32)
    one = _case(None, mode, dtype, 1, 1, rows, hidden, window, layout, autocast)
    cost = work(one)
    room = min(_MOST_FLOPS / cost["flops"], _MOST_BYTES / cost["bytes"])   # (one head alone never exceeds either)
    lots = _log_between(rng, 1, max(1, min(1024, int(room))))
    heads = min(lots, rng.choice([1, 4, 8, 12, 16]))
    return dict(one, batch=max(1, lots // heads), heads=heads)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def prepare(case, seed):
    B, H, M, N = case["batch"], case["heads"], case["rows"], case["hidden"]
    dtype, g = _DTYPES[case["dtype"]], _generator(seed)
    train = case["mode"] != "forward"
    # attention inputs are N(0,1) (the softmax brings the 1/sqrt(N)), those of the bare chain N(0,1)/sqrt(N)
    size = 1.0 if case["mode"] != "chain" else 1.0 / math.sqrt(N)
    shape = (B, M, H * N) if case["layout"] == "proj" else (B, H, M, N)

    def leaf(dims):
        return (torch.randn(dims, device="cuda", generator=g) * size).to(dtype).requires_grad_(train)

    state = {"case": case, "q": leaf(shape), "k": leaf((B, H, N, M) if case["layout"] == "bnm" else shape), "v": leaf(shape)}
    if train:
        out_dtype = torch.float16 if case["autocast"] else dtype
        state["grad_out"] = torch.randn((B, H, M, N), device="cuda", generator=g).to(out_dtype)
    return state


def run(state):
    case = state["case"]
    B, H, M, N, w = case["batch"], case["heads"], case["rows"], case["hidden"], case["window"]
    q, k, v = state["q"], state["k"], state["v"]
    train = case["mode"] != "forward"
    with contextlib.ExitStack() as stack:
        if not train:
            stack.enter_context(torch.no_grad())
        if case["autocast"]:
            stack.enter_context(torch.autocast("cuda", dtype=torch.float16))
        if case["layout"] == "proj":
            qh, kh, vh = (t.view(B, M, H, N).transpose(1, 2) for t in (q, k, v))
        else:
            qh, kh, vh = q, k, v
        keys = kh if case["layout"] == "bnm" else kh.transpose(-1, -2)
        band = window_matmul(qh, keys, w)
        if case["mode"] != "chain":
            band = window_softmax(band, 1.0 / math.sqrt(N))
        out = unwindow_matmul(band, vh, w)
    if not train:
        return {"out": out}
    grad_q, grad_k, grad_v = torch.autograd.grad(out, (q, k, v), state["grad_out"])
    return {"out": out.detach(), "grad_q": grad_q, "grad_k": grad_k, "grad_v": grad_v}


def work(case):
    """Every operator reads its inputs once and writes its outputs once; the band between two operators is an output of
    one and an input of the next.  Under autocast the float32 operands are read, and their gradients written, as such."""
    rows = case["batch"] * case["heads"] * case["rows"]
    wide, band = rows * case["hidden"], rows * (2 * case["window"] + 1)
    size = 4 if case["dtype"] == "float32" and not case["autocast"] else 2
    if case["mode"] == "forward":
        operands, bands, products = 4, 2, 2       # q k -> band; band v -> out
    else:
        operands, bands, products = 11, 5, 6      # ... and q k gband -> gq gk; band v gout -> gband gv
    if case["mode"] != "chain":
        bands += 2 if case["mode"] == "forward" else 5   # softmax: band -> band; backward two bands -> one
    extra = 0
    if case["autocast"]:
        extra = 2 * wide * (3 if case["mode"] == "forward" else 6)
    return {"bytes": size * (operands * wide + bands * band) + extra, "flops": 2 * products * band * case["hidden"]}


def tolerance(case):
    # Measured against the same pass in float64: bfloat16 up to 4.9e-3, float16 up to 6.1e-4 (both: the rounded bands between
    # the operators), float32 up to 5.2e-7 (sums of up to 1025 terms)
    if case["dtype"] == "float16" or case["autocast"]:
        return {"rel": 2.5e-3}
    return {"rel": 5e-6} if case["dtype"] == "float32" else {"rel": 1e-2}
