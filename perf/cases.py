"""Performance cases: what programs built on this framework have it do, through its public entry points.

A case is a dict of plain values.  `op` names the kind of work:

  encoder   the four masked GEMMs of one transformer encoder layer (QKV, attention output, FFN1 with GELU, FFN2
            fed by FFN1), K-major activations, bias fused, output buffers kept by the caller
  gemm      one masked GEMM of a layer on K-major activations
  linear    `A @ (W * mask)` on row-major activations (`masked_linear`)
  tew       a tile-wise layer plus its element-wise residual (`TEWLayer`)
  conv      a pruned stride-1 convolution with bias and ReLU, NHWC in and out (`ConvTWLayer.forward`)
  stream    the reference-signature call, index lists and compacted weights in the caller's hands
  mask      mask construction for a group of layers under one threshold (`build_mask`)
  reprune   one step of gradual pruning: new mask from the scores, the layer re-tiled and re-packed, one forward

Masks are built from the weights with the library's own builder, as a pruning program does; weights and activations
are normal, convolution inputs are non-negative (they follow a ReLU).  Everything is drawn from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import tilesparsity_b200 as ts
from tilesparsity_b200 import masks, stream_gemm, synth, tiles

_DTYPE = {"f16": torch.float16, "bf16": torch.bfloat16}
G = 128     # columns per tile, the width the reference and this framework use throughout


def listed():
    return [
        # One short sequence through an encoder layer (hidden 768, FFN 3072): four calls whose cost is latency.
        {"name": "encoder_m32", "op": "encoder", "M": 32, "hidden": 768, "ffn": 3072, "sparsity": 75.0, "dtype": "f16"},
        # The same layer at the batch the repository's headline is quoted on (32 sequences of 128 tokens).
        {"name": "encoder_m4096", "op": "encoder", "M": 4096, "hidden": 768, "ffn": 3072, "sparsity": 75.0, "dtype": "f16"},
        # The gate matrix of an LSTM translation model over a whole batch of sequences (128 x 50 steps); the result
        # is a new tensor, as in a training or evaluation loop.
        {"name": "lstm_gates", "op": "gemm", "M": 6400, "K": 2048, "N": 4096, "sparsity": 75.0, "dtype": "f16",
         "skew": False, "keep_out": False, "bias": False, "act": ""},
        # The largest single matrix in use: tiles with very different numbers of kept rows.
        {"name": "square_16384", "op": "gemm", "M": 16384, "K": 16384, "N": 16384, "sparsity": 75.0, "dtype": "bf16",
         "skew": True, "keep_out": True, "bias": False, "act": ""},
        # Row-major activations with an odd number of rows, moderate sparsity: the framework's drop-in for a dense
        # `x @ (w * mask)`.
        {"name": "linear_rows", "op": "linear", "M": 3080, "K": 3072, "N": 768, "sparsity": 50.0, "dtype": "bf16"},
        # The LSTM gates with 1.5 % single weights on top of the tiles.
        {"name": "lstm_tew", "op": "tew", "M": 6400, "K": 2048, "N": 4096, "sparsity": 75.0, "extra": 1.5, "dtype": "f16"},
        # A late convolution of an image classifier: small images, many channels, output channels pruned too.
        {"name": "conv_late", "op": "conv", "B": 64, "H": 14, "W": 14, "cin": 512, "cout": 512, "kh": 3, "kw": 3,
         "algo": "tw2", "sparsity": 75.0, "dtype": "bf16"},
        # An early convolution of the same network: large images, few channels.
        {"name": "conv_early", "op": "conv", "B": 8, "H": 112, "W": 112, "cin": 64, "cout": 128, "kh": 3, "kw": 3,
         "algo": "tw1", "sparsity": 50.0, "dtype": "f16"},
        # The reference driver's own call at its published size: half the columns and half the rows kept.
        {"name": "stream_readme", "op": "stream", "M": 12800, "N": 3072, "K": 768, "n_pruned": 1536, "k_pruned": 384, "dtype": "f16"},
        # The mask of one feed-forward matrix: a single small layer.
        {"name": "mask_one", "op": "mask", "group": "one", "K": 768, "N": 3072, "algo": "tw1", "sparsity": 75.0},
        # All convolution kernels of a 13-layer image classifier under one threshold.
        {"name": "mask_group", "op": "mask", "group": "convs", "K": 64, "N": 512, "algo": "tw2", "sparsity": 75.0},
        # A pruning step in a training loop: mask, re-tile, re-pack, forward.
        {"name": "reprune_ffn", "op": "reprune", "M": 4096, "K": 768, "N": 3072, "sparsity": 75.0, "dtype": "f16"},
    ]


def _log(rng, lo, hi, step):
    """A multiple of `step` between lo and hi, uniform over its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / step) * step)))


def draw(rng):
    op = rng.choice(["encoder", "encoder", "gemm", "gemm", "gemm", "linear", "tew", "conv", "conv", "stream", "mask", "mask", "reprune"])
    dtype = rng.choice(["f16", "bf16"])
    sparsity = rng.choice([50.0, 60.0, 75.0, 80.0, 90.0])
    if op == "encoder":
        hidden = rng.choice([256, 384, 512, 768, 1024])
        return {"op": op, "M": _log(rng, 8, 16384, 8), "hidden": hidden, "ffn": 4 * hidden, "sparsity": sparsity, "dtype": dtype}
    if op == "gemm":
        return {"op": op, "M": _log(rng, 8, 16384, 8), "K": _log(rng, 128, 8192, rng.choice([8, 128])),
                "N": _log(rng, 128, 8192, rng.choice([8, 128])), "sparsity": sparsity, "dtype": dtype,
                "skew": rng.random() < 0.3, "keep_out": rng.random() < 0.6, "bias": rng.random() < 0.5,
                "act": rng.choice(["", "", "relu", "gelu"])}
    if op == "linear":
        return {"op": op, "M": _log(rng, 8, 16384, 8), "K": _log(rng, 128, 4096, 8), "N": _log(rng, 128, 4096, 8),
                "sparsity": sparsity, "dtype": dtype}
    if op == "tew":
        return {"op": op, "M": _log(rng, 64, 8192, 8), "K": _log(rng, 256, 4096, 8), "N": _log(rng, 256, 4096, 128),
                "sparsity": rng.choice([60.0, 75.0, 85.0]), "extra": rng.choice([1.0, 1.5, 3.0]), "dtype": dtype}
    if op == "conv":
        side = _log(rng, 7, 112, 1)
        cin, cout = _log(rng, 16, 512, 8), _log(rng, 32, 512, 8)
        k = rng.choice([1, 3, 3, 3, 5])
        most = max(1, min(64, int(1.2e6 / (side * side)), int(4e8 / (side * side * cin))))
        return {"op": op, "B": rng.randint(1, most), "H": side, "W": max(5, side + rng.randint(-2, 2)), "cin": cin, "cout": cout,
                "kh": k, "kw": k, "algo": rng.choice(["tw1", "tw2"]), "sparsity": rng.choice([50.0, 60.0, 75.0]), "dtype": dtype}
    if op == "stream":
        n = _log(rng, 256, 4096, 8)
        k = _log(rng, 128, 4096, 8)
        # (no tile may keep more columns than the N // tiles it owns: whole tiles of kept columns, at most half of N)
        n_pruned = max(G, int(n * rng.uniform(0.3, 0.5)) // G * G)
        return {"op": op, "M": _log(rng, 64, 12800, 8), "N": n, "K": k, "n_pruned": n_pruned,
                "k_pruned": max(8, int(k * rng.uniform(0.1, 0.6)) // 8 * 8), "dtype": dtype}
    if op == "mask":
        return {"op": op, "group": rng.choice(["one", "one", "encoder", "convs"]), "K": _log(rng, 64, 4096, 8), "N": _log(rng, 128, 4096, 8),
                "algo": rng.choice(["tw1", "tw1", "tw2", "tw1m"]), "sparsity": rng.choice([50.0, 75.0, 90.0])}
    return {"op": op, "M": _log(rng, 128, 8192, 8), "K": _log(rng, 256, 4096, 8), "N": _log(rng, 256, 4096, 8),
            "sparsity": sparsity, "dtype": dtype}


# ------------------------------------------------------------------------------------------------ sizes
def _encoder_shapes(case):
    h, f = case["hidden"], case["ffn"]
    return {"qkv": (h, 3 * h), "attn_out": (h, h), "ffn1": (h, f), "ffn2": (f, h)}


def _mask_shapes(case):
    """The score matrices of a mask case, at most 13."""
    k, n = case["K"], case["N"]
    if case["group"] == "one":
        return [(k, n)]
    if case["group"] == "encoder":      # the weight matrices of three encoder layers of hidden size ~ min(K, 1024)
        h = max(128, min(1024, k // 8 * 8))
        return [(h, 3 * h), (h, h), (h, 4 * h), (4 * h, h)] * 3
    # the 13 kernels of a VGG16-shaped network, first stage K channels wide, last stages N wide
    c1, c5 = max(16, min(64, k)), max(128, min(512, n // 8 * 8))
    c = [c1, c1, 2 * c1, 2 * c1, 4 * c1, 4 * c1, 4 * c1, c5, c5, c5, c5, c5, c5]
    return [((3 if i == 0 else c[i - 1]) * 9, c[i]) for i in range(13)]


def work(case):
    """Inputs read once, outputs written once; kept multiply-adds."""
    op = case["op"]
    keep = 1.0 - case["sparsity"] / 100.0 if "sparsity" in case else None

    def gemm(m, k, n, kept):
        return 2.0 * (m * k + m * n + kept), 2.0 * m * kept

    if op == "encoder":
        parts = [gemm(case["M"], k, n, k * n * keep) for k, n in _encoder_shapes(case).values()]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if op in ("gemm", "linear"):
        b, f = gemm(case["M"], case["K"], case["N"], case["K"] * case["N"] * keep)
        return {"bytes": b, "flops": f}
    if op == "tew":
        kept = case["K"] * case["N"] * (keep + case["extra"] / 100.0)
        b, f = gemm(case["M"], case["K"], case["N"], kept)
        return {"bytes": b, "flops": f}
    if op == "conv":
        px = case["B"] * case["H"] * case["W"]
        kept = case["kh"] * case["kw"] * case["cin"] * case["cout"] * keep
        return {"bytes": 2.0 * (px * (case["cin"] + case["cout"]) + kept), "flops": 2.0 * px * kept}
    if op == "stream":
        kept = case["n_pruned"] * case["k_pruned"]
        return {"bytes": 2.0 * (case["M"] * (case["K"] + case["n_pruned"]) + kept), "flops": 2.0 * case["M"] * kept}
    if op == "mask":
        elems = sum(k * n for k, n in _mask_shapes(case))
        return {"bytes": 5.0 * elems, "flops": 2.0 * elems}
    # reprune: scores read, mask written, kept weights read (fp32) and packed, then the forward
    elems = case["K"] * case["N"]
    b, f = gemm(case["M"], case["K"], case["N"], elems * keep)
    return {"bytes": 5.0 * elems + 4.0 * elems * keep + b, "flops": f + 2.0 * elems}


def tolerance(case):
    """Masks and lists are whole numbers and exact; 16-bit results of fp32 sums carry the rounding of their type
    (2^-11 and 2^-8 of a value), a little more where a second 16-bit result is computed from the first."""
    if case["op"] == "mask":
        return "exact"
    return {"rel": 2e-3} if case["dtype"] == "f16" else {"rel": 1e-2}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(g, shape, dtype=torch.float32, scale=1.0):
    x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)
    return (x * scale).to(dtype) if scale != 1.0 else x.to(dtype)


def _skewed_weights(g, K, N, seed, keep, dtype):
    """Weights in their 16-bit type and tiles whose kept-row counts are ~ Beta(2, 5): an iteratively pruned matrix."""
    n_tiles = (N + G - 1) // G
    counts = synth.beta_skewed_counts(K, n_tiles, keep, seed)
    r = synth.rng(seed)
    lists = [np.sort(r.permutation(K)[:int(c)]).astype(np.int32) for c in counts]
    W = torch.randn((K, N), generator=g, device="cuda", dtype=dtype) * 0.02
    return W, tiles.tiles_from_lists(K, N, G, lists)


def _layer(g, K, N, sparsity, dtype, algo="tw1"):
    W = _randn(g, (K, N), scale=0.02)
    res = ts.build_mask(algo, [W.abs()], sparsity, G)
    layer = ts.TWLayer(res.tiles[0], dtype, W.device)
    layer.pack(W)
    return layer


def prepare(case, seed):
    op = case["op"]
    g = _gen(seed)
    dt = _DTYPE.get(case.get("dtype"))
    s = {"case": case, "op": op}
    if op == "encoder":
        M = case["M"]
        s["layers"], s["bias"], s["out"] = {}, {}, {}
        for name, (K, N) in _encoder_shapes(case).items():
            s["layers"][name] = _layer(g, K, N, case["sparsity"], dt)
            s["bias"][name] = _randn(g, (N,), scale=0.02)
            s["out"][name] = torch.zeros((N, M), dtype=dt, device="cuda")
        h = case["hidden"]
        s["x"], s["ctx"], s["y"] = (_randn(g, (h, M), dt) for _ in range(3))
    elif op == "gemm":
        K, N, M = case["K"], case["N"], case["M"]
        if case["skew"]:
            W, t = _skewed_weights(g, K, N, seed, 1.0 - case["sparsity"] / 100.0, dt)
            s["layer"] = ts.TWLayer(t, dt, W.device)
            s["layer"].pack(W)
            del W
        else:
            s["layer"] = _layer(g, K, N, case["sparsity"], dt)
        s["x"] = torch.randn((K, M), generator=g, device="cuda", dtype=dt)
        s["out"] = torch.zeros((N, M), dtype=dt, device="cuda") if case["keep_out"] else None
        s["bias"] = _randn(g, (N,), scale=0.02) if case["bias"] else None
        s["act"] = case["act"] or None
    elif op == "linear":
        s["layer"] = _layer(g, case["K"], case["N"], case["sparsity"], dt)
        s["x"] = _randn(g, (case["M"], case["K"]), dt)
    elif op == "tew":
        W = _randn(g, (case["K"], case["N"]), scale=0.05)
        res = ts.build_mask("tw1m", [W.abs()], case["sparsity"], G, case["extra"], want_residual=True)
        s["layer"] = ts.TEWLayer(W, res.tiles[0], res.residuals[0], dt)
        s["x"] = _randn(g, (case["K"], case["M"]), dt)
    elif op == "conv":
        kh, kw, cin, cout = case["kh"], case["kw"], case["cin"], case["cout"]
        W = _randn(g, (kh, kw, cin, cout), scale=math.sqrt(2.0 / (kh * kw * cin)))
        res = ts.build_mask(case["algo"], masks.img2col_forward([W]), case["sparsity"], G)
        s["layer"] = ts.ConvTWLayer(W, res.tiles[0], dt)
        s["x"] = _randn(g, (case["B"], case["H"], case["W"], cin)).clamp_min_(0).to(dt)
        s["bias"] = _randn(g, (cout,), scale=0.02)
    elif op == "stream":
        M, N, K = case["M"], case["N"], case["K"]
        n_ori, n_cal = tiles.reference_partition(N, case["n_pruned"], G)
        k_cal = [case["k_pruned"]] * len(n_cal)
        r = synth.rng(seed)
        s["mask_k"] = [torch.from_numpy(stream_gemm.mask_gen(r, K, k)).cuda() for k in k_cal]
        s["mask_n"] = [torch.from_numpy(stream_gemm.mask_gen(r, o, c)).cuda() for o, c in zip(n_ori, n_cal)]
        first = [int(sum(n_ori[:t])) for t in range(len(n_ori))]
        B = torch.zeros((N, K), dtype=dt, device="cuda")
        for t, c0 in enumerate(first):
            B[c0:c0 + n_cal[t], :k_cal[t]] = _randn(g, (n_cal[t], k_cal[t]), dt, 0.05)
        s["x"] = _randn(g, (K, M), dt)
        s["out"] = torch.zeros((N, M), dtype=dt, device="cuda")
        s["call"] = stream_gemm.prepare_stream_gemm_nn(M, N, K, 1.0, s["x"], B, 0.0, s["out"], len(n_cal), n_cal, k_cal, s["mask_n"],
                                                       s["mask_k"], [K * c for c in first], [M * c for c in first])
    elif op == "mask":
        shapes = _mask_shapes(case)
        s["scores"] = [_randn(g, shape, scale=0.02).abs_() for shape in shapes]
        # where the program keeps the index lists: as long as they can get, for their lengths follow from the scores
        s["lists"] = [[np.full(n + 1, -1, np.int32) for n in ((N + G - 1) // G + 1, K * ((N + G - 1) // G), N)] for K, N in shapes]
    else:
        K, N = case["K"], case["N"]
        s["W"] = _randn(g, (K, N), scale=0.02)
        s["scores"] = s["W"].abs()
        res = ts.build_mask("tw1", [s["scores"]], max(0.0, case["sparsity"] - 10.0), G)   # the structure of the step before
        s["layer"] = ts.TWLayer(res.tiles[0], dt, s["W"].device)
        s["layer"].pack(s["W"])
        s["x"] = _randn(g, (K, case["M"]), dt)
        s["out"] = torch.zeros((N, case["M"]), dtype=dt, device="cuda")
    return s


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    op = state["op"]
    if op == "encoder":
        lay, b, o = state["layers"], state["bias"], state["out"]
        qkv = lay["qkv"].masked_gemm(state["x"], out=o["qkv"], bias=b["qkv"])
        attn = lay["attn_out"].masked_gemm(state["ctx"], out=o["attn_out"], bias=b["attn_out"])
        mid = lay["ffn1"].masked_gemm(state["y"], out=o["ffn1"], bias=b["ffn1"], activation="gelu")
        return [qkv, attn, mid, lay["ffn2"].masked_gemm(mid, out=o["ffn2"], bias=b["ffn2"])]
    if op == "gemm":
        return state["layer"].masked_gemm(state["x"], out=state["out"], bias=state["bias"], activation=state["act"])
    if op == "linear":
        return ts.masked_linear(state["x"], state["layer"])
    if op == "tew":
        return state["layer"].masked_gemm(state["x"])
    if op == "conv":
        return state["layer"].forward(state["x"], bias=state["bias"], activation="relu")
    if op == "stream":
        state["call"]()
        return state["out"]
    if op == "mask":
        c = state["case"]
        res = ts.build_mask(c["algo"], state["scores"], c["sparsity"], G)
        for t, (ptr, rows, cols) in zip(res.tiles, state["lists"]):
            for dst, src in ((ptr, t.tile_k_ptr), (rows, t.kept_k), (cols, t.kept_n)):
                dst[:len(src)] = src
        return {"masks": res.masks, "thresholds": [float(v) for v in res.thresholds], "lists": state["lists"]}
    res = ts.build_mask("tw1", [state["scores"]], state["case"]["sparsity"], G)
    state["layer"].retile(res.tiles[0])
    state["layer"].pack(state["W"])
    out = state["layer"].masked_gemm(state["x"], out=state["out"])
    return {"out": out, "mask": res.masks[0], "kept_k": res.tiles[0].kept_k}
