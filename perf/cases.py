"""The work that a user of this library has it do, as cases that can be timed and compared.

A case is a dict of plain values. ``op`` names the public operator:

* ``flash_attention``: ``B, Hq, Hkv, M, N, D, dtype, causal, layout, train, aux, dropout``. ``train`` adds the backward
  (gradients of q, k and v through autograd), ``aux`` the log-normaliser and the total attention, ``layout`` says
  whether q, k, v are contiguous ``[B, H, T, D]`` tensors or transposed views of a projection's ``[B, T, H, D]`` output.
* ``flash_attention_split_kv``: ``B, Hq, Hkv, M, N, D, dtype, causal``: new tokens against a dense K/V cache.
* ``paged_attention``: ``B`` sequences of different lengths up to ``N`` keys in cache blocks of ``block`` keys.
* ``piecewise_attention``: ``B, Hq, M, N, D, dtype, causal, dist, train``.

Inputs are N(0, 1), the distribution of normalised queries and keys and the one that this repository's tests and
benchmark use. Sizes are those of the benchmark's workloads, of the tests, or generic.
"""
import math
import random

import torch

import flagattention_b200 as fa

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _attn(name, B, Hq, Hkv, M, N, D, dtype, causal, train=False, aux=False, dropout=0.0, layout="BHTD"):
    return {"name": name, "op": "flash_attention", "B": B, "Hq": Hq, "Hkv": Hkv, "M": M, "N": N, "D": D, "dtype": dtype,
            "causal": causal, "layout": layout, "train": train, "aux": aux, "dropout": dropout}


def listed():
    return [
        # One short prompt through one layer: the latency of a single call.
        _attn("prompt_128_d64", 1, 4, 4, 128, 128, 64, "fp16", False),
        # A training step of a small model on a short sequence: launches and host work count as much as the kernels.
        _attn("train_small_512", 2, 8, 2, 512, 512, 128, "bf16", True, train=True),
        # Many short sequences (encoder-like batch, head dimension 64): a few tiles per work item, prologues count.
        _attn("train_short_d64", 64, 32, 32, 512, 512, 64, "fp16", True, train=True),
        # Odd lengths after a cached prefix, grouped heads, transposed views as they come from a projection.
        _attn("train_ragged_1537", 3, 16, 4, 1111, 1537, 128, "bf16", True, train=True, layout="BTHD"),
        # The grouped-head training step of the benchmark.
        _attn("train_gqa_4096", 4, 32, 8, 4096, 4096, 128, "bf16", True, train=True),
        # Training with dropout and both auxiliary outputs.
        _attn("train_dropout_d64", 16, 16, 16, 2048, 2048, 64, "fp16", False, train=True, aux=True, dropout=0.1),
        # Cross attention of 512 queries over one KV head.
        _attn("cross_mqa_8192", 8, 16, 1, 512, 8192, 128, "bf16", False),
        # Prefill of a long context, the largest call.
        _attn("prefill_32768", 1, 64, 8, 32768, 32768, 128, "bf16", True),
        # One new token per sequence against a dense cache of ordinary length, one query head per KV head.
        {"name": "decode_mha_8192", "op": "flash_attention_split_kv", "B": 2, "Hq": 16, "Hkv": 16, "M": 1, "N": 8192,
         "D": 128, "dtype": "fp16", "causal": False},
        # The same with grouped heads, a larger batch and a long cache.
        {"name": "decode_gqa_32768", "op": "flash_attention_split_kv", "B": 8, "Hq": 32, "Hkv": 8, "M": 1, "N": 32768,
         "D": 128, "dtype": "bf16", "causal": False},
        # A serving batch over a paged cache, every sequence at another length.
        {"name": "paged_gqa_4096", "op": "paged_attention", "B": 32, "Hq": 64, "Hkv": 8, "N": 4096, "D": 128,
         "dtype": "fp16", "block": 16},
        # Two pairs of (q, k) selected by distance (extrapolation beyond the trained length), training step.
        {"name": "piecewise_train_2048", "op": "piecewise_attention", "B": 4, "Hq": 16, "M": 2048, "N": 2048, "D": 128,
         "dtype": "bf16", "causal": True, "dist": 1024, "train": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pairs(M, N, causal):
    """Visible (query, key) pairs; query m sees the keys n <= m + N - M under a causal mask."""
    if not causal:
        return M * N
    d = N - M  # the drawn and listed causal cases have M <= N
    return M * (d + 1) + M * (M - 1) // 2


def draw(rng):
    """One more case of the listed ranges: lengths 64 to 32768 (odd ones too), head dimensions 32, 64 and 128, one
    to eight query heads per KV head, forward and backward, and never more work than the listed cases have."""
    while True:
        op = rng.choice(["train", "train", "train", "forward", "forward", "dropout", "decode", "decode", "paged", "piecewise"])
        D = rng.choice([32, 64, 64, 128, 128, 128])
        dtype = rng.choice(["fp16", "bf16"])
        group = rng.choice([1, 1, 2, 4, 8])
        Hkv = rng.choice([1, 2, 4, 8, 16])
        Hq = Hkv * group
        causal = rng.random() < 0.7
        if op in ("train", "forward"):
            N = _log_int(rng, 64, 32768 if op == "forward" else 8192)
            M = N if rng.random() < 0.5 else _log_int(rng, min(64, N), N)
            B = _log_int(rng, 1, 64)
            case = _attn("", B, Hq, Hkv, M, N, D, dtype, causal, train=op == "train", aux=rng.random() < 0.15,
                         layout=rng.choice(["BHTD", "BTHD"]))
            flops, limit = 4.0 * B * Hq * _pairs(M, N, causal) * D, (8e12 if op == "forward" else 8e11)
            size = B * D * (Hq * M + Hkv * N)
            fits = flops <= limit and size <= 3e8
        elif op == "dropout":
            N = _log_int(rng, 64, 4096)
            B = _log_int(rng, 1, 16)
            p = rng.choice([0.1, 0.2])
            case = _attn("", B, Hq, Hkv, N, N, D, dtype, causal, train=True, aux=rng.random() < 0.3, dropout=p)
            # short calls with few heads take the split-key branch, which has no dropout
            fits = B * Hq * (-(-N // 16)) >= 256 and B * Hq * _pairs(N, N, causal) <= 6e8 and B * D * (Hq + Hkv) * N <= 1e8
        elif op == "decode":
            N, B, M = _log_int(rng, 128, 65536), _log_int(rng, 1, 32), rng.choice([1, 1, 1, 2, 4])
            case = {"op": "flash_attention_split_kv", "B": B, "Hq": Hq, "Hkv": Hkv, "M": M, "N": N, "D": D,
                    "dtype": dtype, "causal": M > 1}
            fits = B * Hkv * N * D <= 2.7e8
        elif op == "paged":
            N, B, D = _log_int(rng, 128, 16384), _log_int(rng, 1, 128), rng.choice([64, 128, 128])
            case = {"op": "paged_attention", "B": B, "Hq": Hq, "Hkv": Hkv, "N": N, "D": D, "dtype": dtype,
                    "block": rng.choice([16, 16, 32, 64, 128])}
            fits = B * Hkv * N * D <= 2.7e8
        else:
            N = _log_int(rng, 128, 4096)
            B = _log_int(rng, 1, 8)
            D = rng.choice([64, 128])
            case = {"op": "piecewise_attention", "B": B, "Hq": Hq, "M": N, "N": N, "D": D, "dtype": dtype, "causal": causal,
                    "dist": max(1, int(N * rng.uniform(0.25, 0.75))), "train": rng.random() < 0.7}
            fits = 4.0 * B * Hq * _pairs(N, N, causal) * D <= 3e11
        case.pop("name", None)
        if fits:
            return case


def _context_lens(case):
    """Key counts of the paged sequences: spread evenly from a quarter of the longest context to all of it."""
    B, N = case["B"], case["N"]
    return [N - (N - -(-N // 4)) * i // max(1, B - 1) for i in range(B)]


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    dtype = _DTYPES[case["dtype"]]
    gen = torch.Generator(device=dev).manual_seed(seed)

    def normal(*shape):
        return torch.randn(shape, generator=gen, device=dev, dtype=dtype)

    op, D = case["op"], case["D"]
    if op == "paged_attention":
        # The scheduler of a serving program knows every length, so the largest one costs no read-back.
        lens = _context_lens(case)
        random.Random(seed).shuffle(lens)
        block, Hkv = case["block"], case["Hkv"]
        counts = [-(-n // block) for n in lens]
        num_blocks, widest = sum(counts), max(counts)
        perm = torch.randperm(num_blocks, generator=gen, device=dev).to(torch.int32)
        tables = torch.zeros(case["B"], widest, dtype=torch.int32, device=dev)
        start = 0
        for i, n in enumerate(counts):
            tables[i, :n] = perm[start:start + n]
            start += n
        return {"op": op, "q": normal(case["B"], case["Hq"], D), "k": normal(num_blocks, Hkv, block, D),
                "v": normal(num_blocks, Hkv, block, D), "lens": torch.tensor(lens, dtype=torch.int32, device=dev),
                "tables": tables, "scale": 1.0 / math.sqrt(D), "longest": max(lens)}

    def heads(H, T):
        if case.get("layout") == "BTHD":
            return normal(case["B"], T, H, D).transpose(1, 2)
        return normal(case["B"], H, T, D)

    Hq, M, N = case["Hq"], case["M"], case["N"]
    state = {"op": op, "causal": case["causal"]}
    if op == "flash_attention_split_kv":
        state.update(inputs=(heads(Hq, M), heads(case["Hkv"], N), heads(case["Hkv"], N)))
        return state
    if op == "piecewise_attention":
        inputs = (heads(Hq, M), heads(Hq, N), heads(Hq, M), heads(Hq, N), heads(Hq, N))
        state.update(dist=case["dist"])
    else:
        inputs = (heads(Hq, M), heads(case["Hkv"], N), heads(case["Hkv"], N))
        state.update(aux=case["aux"], dropout=case["dropout"], seed=seed)
    state.update(inputs=inputs, d_out=None)
    if case["train"]:
        for t in inputs:
            t.requires_grad_()
        state["d_out"] = heads(Hq, M)
    return state


def run(state):
    op = state["op"]
    if op == "paged_attention":
        return fa.paged_attention(state["q"], state["k"], state["v"], state["lens"], state["tables"], state["scale"],
                                  state["longest"])
    inputs, causal = state["inputs"], state["causal"]
    if op == "flash_attention_split_kv":
        return fa.flash_attention_split_kv(*inputs, causal=causal)
    if op == "piecewise_attention":
        out = fa.piecewise_attention(*inputs, state["dist"], causal=causal)
        outputs = (out,)
    else:
        if state["dropout"] > 0:
            torch.cuda.manual_seed(state["seed"])  # a reproducible step: every pass over a state draws the same mask
        result = fa.flash_attention(*inputs, causal=causal, dropout_p=state["dropout"],
                                    return_log_normalizer=state["aux"], return_total_attention=state["aux"])
        out = result[0] if state["aux"] else result
        outputs = (out,) + (result[1:3] if state["aux"] else ())
    if state["d_out"] is not None:
        outputs += torch.autograd.grad(out, inputs, state["d_out"])
    return outputs


def work(case):
    """Every input read once, every output written once, and the products over the visible pairs: two in the forward,
    five in the backward, one more for the total attention (it needs the finished log-normaliser)."""
    op, D = case["op"], case["D"]
    if op == "paged_attention":
        keys = sum(_context_lens(case))
        return {"bytes": 2 * D * (2 * case["Hkv"] * keys + 2 * case["B"] * case["Hq"]), "flops": 4.0 * case["Hq"] * keys * D}
    B, Hq, M, N = case["B"], case["Hq"], case["M"], case["N"]
    Hkv = case.get("Hkv", Hq)
    train, pair = case.get("train", False), op == "piecewise_attention"
    q_side, kv_side = B * Hq * M * D, B * Hkv * N * D
    n_q, n_kv = (2, 3) if pair else (1, 2)
    elements = (n_q + 1) * q_side + n_kv * kv_side                    # q.., k.., v in, o out
    if train:
        elements += (n_q + 1) * q_side + n_kv * kv_side               # dO in, the gradients out
    units = 2.0 + (5.0 if train else 0.0) + (1.0 if case.get("aux") else 0.0)
    aux = 4 * B * Hq * (M + N) if case.get("aux") else 0
    return {"bytes": 2 * elements + aux, "flops": 2.0 * units * B * Hq * _pairs(M, N, case["causal"]) * D}


def tolerance(case):
    """Four times what these operators show against the same attention in float64: 2.5e-3 (2-norm) and 0.1 (largest
    element) with bf16 operands, whose probabilities and results are rounded to 8 bits, 3.1e-4 and 0.012 with fp16."""
    return {"rel": 1e-2, "max": 0.4} if case["dtype"] == "bf16" else {"rel": 1.2e-3, "max": 0.05}
