"""The host fast path, the row-major and NHWC outputs, re-tiling and the grouped mask stages, at the sizes where each
changes form.  GEMM results against float64 products of the same 16-bit inputs: the fp32 accumulation over K <= 3072
rounds far below the 16-bit result, whose half unit is 2^-11 (fp16) or 2^-8 (bf16) of a value; TOL below is four
times that, as a 2-norm ratio."""
import ctypes as C
import gc
import threading

import numpy as np
import pytest
import torch

from oracle import tw_masks as om
from tilesparsity_b200 import synth

pytestmark = pytest.mark.gpu
TOL = {torch.float16: 2e-3, torch.bfloat16: 1.6e-2}


def _layer(K, N, keep, dtype, seed, col_keep=None):
    from tilesparsity_b200 import TWLayer
    g = synth.rng(seed)
    col = (g.random(N) < col_keep) if col_keep is not None else None
    from tilesparsity_b200.tiles import tile_bounds_from_col_mask
    nt = len(tile_bounds_from_col_mask(np.ones(N, bool) if col is None else col, 128)) - 1
    lists = [np.sort(g.permutation(K)[:keep]).astype(np.int32) for _ in range(nt)]
    W = torch.from_numpy(g.standard_normal((K, N), dtype=np.float32) * np.float32(0.05)).cuda()
    return TWLayer.from_lists(W, lists, col, 128, dtype), W


def _dense(W, layer, dtype):
    """W .* mask in float64, from the 16-bit weights."""
    mask = torch.from_numpy(layer.tiles.dense_mask()).to(W.device)
    return W.to(dtype).double() * mask


def _rel(out, ref):
    return float((out.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,K,N,col_keep", [
    (8, 64, 128, None),           # one tile, eight rows
    (64, 256, 136, None),         # a last tile of eight columns
    (72, 256, 248, None),         # a last tile of 120 columns: its last warp's box is cut off
    (3080, 768, 768, None),       # odd numbers of granules, three per SM
    (1000, 3072, 1536, None),
    (264, 260, 204, None),        # N not a multiple of eight: output transposed back, two-byte transposes
    (520, 512, 640, 0.7),         # pruned columns: output transposed back, zeros in them
])
def test_row_major_linear(M, K, N, col_keep, dtype):
    from tilesparsity_b200 import masked_linear
    layer, W = _layer(K, N, max(8, K // 3), dtype, M + K + N, col_keep)
    A = torch.randn((M, K), device="cuda", generator=torch.Generator("cuda").manual_seed(M)).to(dtype)
    torch.empty((64 << 20,), dtype=torch.uint8, device="cuda").fill_(0x7f)     # what the allocator hands out next is not zero
    ref = A.double() @ _dense(W, layer, dtype)
    C = masked_linear(A, layer)
    layer.check()
    assert C.shape == (M, N) and C.is_contiguous() and _rel(C, ref) <= TOL[dtype]
    Ct = masked_linear(A, layer, transpose_out=False)
    assert Ct.shape == (N, M) and torch.equal(Ct.t(), C)
    dead = torch.from_numpy(~layer.tiles.col_mask()).cuda()
    assert not C[:, dead].any()
    layer.close()


def test_row_major_linear_takes_a_tew_layer():
    from tilesparsity_b200 import TEWLayer, build_mask, masked_linear
    W = torch.randn((256, 384), device="cuda", generator=torch.Generator("cuda").manual_seed(1)) * 0.05
    res = build_mask("tw2m", [W.abs()], 60.0, 128, 2.0, want_residual=True)
    layer = TEWLayer(W, res.tiles[0], res.residuals[0], torch.float16)
    A = torch.randn((72, 256), device="cuda").half()
    ref = A.double() @ (W.half().double() * res.masks[0])
    assert _rel(masked_linear(A, layer), ref) <= TOL[torch.float16]
    # columns without any kept element are cleared in a caller's buffer
    out = torch.full((384, 72), float("nan"), dtype=torch.float16, device="cuda")
    assert _rel(layer.masked_gemm(A.t().contiguous(), out=out).t(), ref) <= TOL[torch.float16]
    layer.close()


@pytest.mark.parametrize("rows,cols,skip", [(8, 8, 0), (128, 136, 0), (120, 1024, 8), (1, 8, 0), (130, 250, 0), (136, 264, 4)])
def test_transpose(rows, cols, skip):
    """skip: the view starts that many elements into a wider matrix (16-byte pieces only where it is a multiple of 8)."""
    from tilesparsity_b200 import transpose16
    x = torch.randint(-32768, 32767, (rows, cols + skip), dtype=torch.int16, device="cuda")[:, skip:]
    assert torch.equal(transpose16(x), x.t())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("col_keep", [None, 0.8])
def test_new_outputs_are_whole(dtype, col_keep):
    """An output the call makes itself: every kept column written, every pruned one zero, whatever its memory held."""
    layer, W = _layer(128, 520, 40, dtype, 11, col_keep)
    At = torch.randn((128, 264), device="cuda").to(dtype)
    ref = _dense(W, layer, dtype).t() @ At.double()
    for _ in range(3):
        junk = torch.full((520, 264), float("nan"), dtype=dtype, device="cuda")
        del junk
        out = layer.masked_gemm(At)
        assert _rel(out, ref) <= TOL[dtype]
        assert not out[torch.from_numpy(~layer.tiles.col_mask()).cuda()].any()
    layer.close()


@pytest.mark.parametrize("col_keep", [None, 0.8])
def test_gelu_at_the_ends_of_the_range(col_keep):
    """The tanh form's limits: 0 for large negative sums (whatever their neighbours), the sum itself for large positive
    ones, NaN for NaN and for -inf.  Bias carries the values: eight batch rows of zeros."""
    layer, _ = _layer(64, 256, 16, torch.bfloat16, 5, col_keep)
    vals = [-1e30, 1e30, -1e30, -1e30, -50.0, 50.0, -7.9, 0.5, float("inf"), -3e38, float("nan"), -1.0, float("-inf"), 2.0]
    bias = torch.tensor((vals * 19)[:256], device="cuda")
    out = layer.masked_gemm(torch.zeros((64, 72), dtype=torch.bfloat16, device="cuda"), bias=bias, activation="gelu")
    x = bias.double()
    ref = x * 0.5 * (1 + torch.tanh((2 / np.pi) ** 0.5 * (x + 0.044715 * x ** 3)))
    kept = torch.from_numpy(layer.tiles.col_mask()).cuda()
    got, want = out.double()[kept], ref[kept, None].expand(-1, 72)
    assert torch.equal(got.isnan(), want.isnan())
    ok = ~want.isnan()
    # (bf16 rounding, and 1e-12 where the tanh form in any precision cancels to nothing)
    assert torch.allclose(got[ok], want[ok], rtol=2 ** -8, atol=1e-12)
    layer.close()


def test_outputs_that_alternate_and_threads():
    """More output buffers than the layer remembers, from four threads with a stream each."""
    layer, W = _layer(256, 512, 100, torch.float16, 9)
    x = torch.randn((256, 520), device="cuda").half()
    ref = layer.masked_gemm(x)
    outs = [[torch.zeros_like(ref) for _ in range(6)] for _ in range(4)]
    torch.cuda.synchronize()
    errors = []

    def work(mine):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                for _ in range(20):
                    for o in mine:
                        layer.masked_gemm(x, out=o)
            s.synchronize()
        except Exception as e:      # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(m,)) for m in outs]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors
    assert all(torch.equal(o, ref) for m in outs for o in m)
    layer.close()


def test_an_output_that_cannot_be_allocated_is_an_error():
    layer, _ = _layer(64, 8192, 16, torch.float16, 2)
    x = torch.zeros((64, 8), dtype=torch.float16, device="cuda")
    before = layer.masked_gemm(x)
    with pytest.raises(torch.cuda.OutOfMemoryError):
        layer.masked_gemm(torch.empty((64, 1 << 24), dtype=torch.float16, device="cuda"))    # 275 GB of output
    assert torch.equal(layer.masked_gemm(x), before)
    layer.close()


def _stream_case(M, N, K, n_pruned, k_pruned, seed):
    from tilesparsity_b200 import stream_gemm, tiles
    r = synth.rng(seed)
    n_ori, n_cal = tiles.reference_partition(N, n_pruned, 128)
    first = [int(sum(n_ori[:t])) for t in range(len(n_ori))]
    k_cal = [k_pruned] * len(n_cal)
    mk = [stream_gemm.mask_gen(r, K, k) for k in k_cal]
    mn = [stream_gemm.mask_gen(r, o, c) for o, c in zip(n_ori, n_cal)]
    B = torch.zeros((N, K), dtype=torch.float16, device="cuda")
    A = torch.randn((K, M), device="cuda").half()
    ref = torch.zeros((N, M), dtype=torch.float64, device="cuda")
    for t, c0 in enumerate(first):
        w = torch.randn((n_cal[t], k_pruned), device="cuda").half() * 0.05
        B[c0:c0 + n_cal[t], :k_pruned] = w
        rows = torch.from_numpy(mk[t] + np.arange(k_pruned)).cuda().long()
        cols = torch.from_numpy(mn[t] + np.arange(n_cal[t]) + c0).cuda().long()
        ref[cols] = w.double() @ A[rows].double()
    C = torch.zeros((N, M), dtype=torch.float16, device="cuda")
    call = stream_gemm.prepare_stream_gemm_nn(M, N, K, 1.0, A, B, 0.0, C, len(n_cal), n_cal, k_cal, [torch.from_numpy(m).cuda() for m in mn],
                                              [torch.from_numpy(m).cuda() for m in mk], [K * c for c in first], [M * c for c in first])
    return call, C, ref


def test_stream_calls_share_schedules_by_shape():
    """Same shape with other lists and buffers, and more shapes than are kept: every call uses its own lists.  A graph's
    schedule outlives them."""
    cases = [_stream_case(264, 512, 256, 256, 64, s) for s in (1, 2)]
    graph = torch.cuda.CUDAGraph()
    cases[0][0]()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        cases[0][0]()
    cases += [_stream_case(8 * m, 384, 128, 256, 40, m) for m in range(1, 20)]
    for _ in range(2):
        for call, C, ref in cases:
            C.fill_(0)
            call()
            assert _rel(C, ref) <= TOL[torch.float16]
    cases[0][1].fill_(0)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert _rel(cases[0][1], cases[0][2]) <= TOL[torch.float16]


@pytest.mark.parametrize("algo,sparsity,shapes", [
    ("tw1", 75.0, [(128, 128 * 128)]),                       # 16384 tile rows: one block's percentile
    ("tw1", 75.0, [(129, 128 * 128)]),                       # 16512: a cluster's
    ("tw1", np.float64(60.0), [(1100, 128 * 128)]),          # more lists than fit the page-locked block
    ("tw1", 50.0, [(40 + i, 136 + 8 * (i % 5)) for i in range(41)]),      # more layers than the kernel arguments hold
    ("tw2", 70.0, [(33 + i, 100 + 7 * (i % 9)) for i in range(41)]),
    ("tw2", 0.0, [(64, 256), (70, 130)]),                    # nothing pruned but the minimum
    ("tw2", 99.0, [(64, 300)]),                              # tiles without rows
    ("tw1m", 75.0, [(1025, 1024)]),                          # residual: more values than a cluster ranks
])
def test_grouped_masks_match_oracle(algo, sparsity, shapes):
    from tilesparsity_b200 import build_mask
    g = np.random.Generator(np.random.PCG64(len(shapes) * 1000 + shapes[0][0]))
    scores = [np.abs(g.standard_normal(s, dtype=np.float32)) for s in shapes]
    ref = om.pruning_fun(algo)(scores, sparsity, 128)
    dev = [torch.from_numpy(s).cuda() for s in scores]
    dev[0] = torch.nn.functional.pad(dev[0], (0, 3))[:, :dev[0].shape[1]]        # a row pitch that allows no 16-byte loads
    res = build_mask(algo, dev, sparsity, 128, want_residual=algo.endswith("m"))
    for l, (m, r) in enumerate(zip(res.masks, ref)):
        r = np.asarray(r, dtype=bool)
        assert np.array_equal(m.cpu().numpy(), r), l
        if not algo.endswith("m"):
            assert np.array_equal(res.tiles[l].dense_mask(), r), l


@pytest.mark.parametrize("algo,sparsity", [("tw1", 75.0), ("tw1", np.float64(60.0)), ("tw2", 50.0), ("tw2", 99.0), ("bert_type8", 30.0)])
def test_groups_of_more_than_a_million_tile_rows_match_oracle(algo, sparsity):
    """Beyond what one cluster ranks (2^20 norms): two layers, tiles of 8 columns.  At 99 % the columns that are left make
    fewer norms than that."""
    from tilesparsity_b200 import build_mask
    g = np.random.Generator(np.random.PCG64(77))
    scores = [np.abs(g.standard_normal(s, dtype=np.float32)) for s in ((900, 8192), (400, 4096))]
    ref = om.pruning_fun(algo)(scores, sparsity, 8) if algo != "bert_type8" else om.bert_type8(scores, sparsity, 8)
    res = build_mask(algo, [torch.from_numpy(s).cuda() for s in scores], sparsity, 8)
    for l, (m, r) in enumerate(zip(res.masks, ref)):
        r = np.asarray(r, dtype=bool)
        assert np.array_equal(m.cpu().numpy(), r), l
        assert np.array_equal(res.tiles[l].dense_mask(), r), l


@pytest.mark.parametrize("B,H,W,cin,cout,kh,kw,algo", [
    (2, 5, 7, 16, 40, 3, 3, "tw1"),        # one narrow tile; two blocks of 8 channels in, five out
    (3, 14, 14, 72, 256, 3, 3, "tw1"),     # nine blocks of channels in: no lane layout but one or two fits
    (1, 9, 20, 24, 136, 5, 3, "tw1"),      # a second tile of eight channels
    (2, 1, 1, 8, 8, 1, 1, "tw1"),          # one pixel
    (5, 3, 260, 64, 128, 1, 5, "tw1"),     # rows of many groups
    (3, 14, 14, 64, 264, 3, 3, "tw2"),     # pruned channels: through the padded space
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_convolution_output_forms_agree(B, H, W, cin, cout, kh, kw, algo, dtype):
    """forward (NHWC from the GEMM where the tiles allow it) == GEMM into the padded space + unpacking, bit for bit, and
    == conv2d in float64."""
    from tilesparsity_b200 import ConvTWLayer, build_mask, masks
    g = torch.Generator("cuda").manual_seed(B * 1000 + W)
    w = torch.randn((kh, kw, cin, cout), device="cuda", generator=g) * (2.0 / (kh * kw * cin)) ** 0.5
    res = build_mask(algo, masks.img2col_forward([w]), 40.0, 128)
    layer = ConvTWLayer(w, res.tiles[0], dtype)
    x = torch.randn((B, H, W, cin), device="cuda", generator=g).to(dtype)
    bias = torch.randn((cout,), device="cuda", generator=g)
    junk = torch.full((B, H, W, cout), float("nan"), dtype=dtype, device="cuda")
    del junk
    y = layer.forward(x, bias=bias, activation="relu")
    planes, geo = layer.pack_input(x)
    padded = layer.masked_conv(planes, geo, out=torch.zeros((cout, geo["m_padded"]), dtype=dtype, device="cuda"), bias=bias,
                               activation="relu")
    layer.layer.check()
    assert torch.equal(y, layer.unpack_output(padded, geo))
    wm = (w.to(dtype).double() * res.masks[0].view(kh, kw, cin, cout)).permute(3, 2, 0, 1)
    ref = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), wm, bias.double(), padding=(kh // 2, kw // 2)).clamp_min(0)
    kept = torch.from_numpy(res.tiles[0].col_mask()).cuda()
    ref = ref.permute(0, 2, 3, 1) * kept
    assert _rel(y, ref) <= TOL[dtype]
    layer.close()


def test_retiling_reuses_memory_soundly():
    """A layer re-tiled between products, larger and smaller, and products of more batch sizes than schedules are kept
    (split-K ones among them): every product is that of its own tiles."""
    from tilesparsity_b200 import TWLayer, tiles
    K, N = 4096, 256
    W = torch.randn((K, N), device="cuda") * 0.05
    layer = None
    for step, keep in enumerate([3000, 500, 2600, 64, 4096, 200]):
        g = synth.rng(step)
        t = tiles.tiles_from_lists(K, N, 128, [np.sort(g.permutation(K)[:keep]).astype(np.int32) for _ in range(2)])
        if layer is None:
            layer = TWLayer(t, torch.float16, W.device)
        else:
            layer.retile(t)
        layer.pack(W)
        Wm = _dense(W, layer, torch.float16)
        for M in [8 * m for m in range(1, 19)] + [2048]:
            x = torch.randn((K, M), device="cuda").half()
            assert _rel(layer.masked_gemm(x), Wm.t() @ x.double()) <= TOL[torch.float16]
    layer.check()
    layer.close()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("algo,K,N,M,alpha", [
    ("tw1m", 256, 384, 64, 1.0),        # full tiles
    ("tw2m", 250, 300, 1032, 0.5),      # pruned columns, K no multiple of eight, a second block of batch rows
    ("tw1m", 4096, 128, 64, 1.0),       # long chains: split-K
    ("tw1m", 256, 8, 8, -2.0),          # one tile of eight columns
])
@pytest.mark.parametrize("everywhere", [False, True])     # one feature infinite, one NaN in every batch row
def test_tew_keeps_non_finite_activations_to_the_columns_that_keep_their_rows(algo, K, N, M, alpha, everywhere, dtype):
    """Infinities and NaN in the activations: every output is what the mask's own entries give (an infinity of that
    sign, NaN where they clash, a finite sum where the column keeps no such row)."""
    from tilesparsity_b200 import TEWLayer, build_mask
    g = torch.Generator("cuda").manual_seed(K + N)
    W = torch.randn((K, N), device="cuda", generator=g) * 0.05
    res = build_mask(algo, [W.abs()], 75.0, 128, 1.5, want_residual=True)
    layer = TEWLayer(W, res.tiles[0], res.residuals[0], dtype)
    kept = res.masks[0] | res.residuals[0]
    x = torch.randn((K, M), device="cuda", generator=g).to(dtype)
    inf = float("inf")
    for k, m, v in [(7, 3, inf), (100, 3, -inf), (101, 5, float("nan")), (K - 1, M - 1, -inf), (0, 0, inf), (3, 0, inf)]:
        x[k, m] = v
    if everywhere:                                       # (features that the fewest columns keep)
        few = [k for k in torch.argsort(kept.sum(1)).tolist() if kept[k].any()]
        x[few[0]], x[few[1]] = inf, float("nan")
        if N == 8:
            x[[0, 3, 7, 100, 101, K - 1]] = 0.5
    ref = torch.zeros((N, M), dtype=torch.float64, device="cuda")
    Wd, xd = W.to(dtype).double(), x.double()
    for n in range(N):
        ref[n] = alpha * (Wd[kept[:, n], n] @ xd[kept[:, n]])
    for out in (None, torch.full((N, M), 7.0, dtype=dtype, device="cuda")):
        got = layer.masked_gemm(x, out=out, alpha=alpha).double()
        assert torch.equal(got.isnan(), ref.isnan())
        assert torch.equal(got.isinf(), ref.isinf()) and torch.equal(got[ref.isinf()], ref[ref.isinf()])
        ok = ref.isfinite()
        assert 0 < int((~ok).sum()) < ref.numel()
        assert float((got[ok] - ref[ok]).norm() / ref[ok].norm()) <= TOL[dtype]
    layer.close()


def test_an_allocation_that_fails_is_reported_once():
    """A tile structure that needs 275 GB of packed weights (nothing is allocated) is an error of that call; the next
    layer's packing and product know nothing of it."""
    from tilesparsity_b200 import TWLayer, _lib, tiles
    K, N = 1 << 19, 1 << 18
    rows = [np.arange(K, dtype=np.int32)] + [np.arange(8, dtype=np.int32)] * (N // 128 - 1)
    with pytest.raises(_lib.TileSparseError):
        TWLayer(tiles.tiles_from_lists(K, N, 128, rows), torch.float16, "cuda")
    layer, W = _layer(64, 128, 16, torch.float16, 3)
    x = torch.randn((64, 8), device="cuda").half()
    assert _rel(layer.masked_gemm(x), _dense(W, layer, torch.float16).t() @ x.double()) <= TOL[torch.float16]
    layer.close()


def test_a_retiling_that_fails_leaves_a_layer_without_tiles():
    """More packed weights than any GPU holds (275 GB; nothing is allocated): the call is an error, and so is every
    product of the layer after it.  New outputs have pruned columns to clear, whose list is gone with the old tiles."""
    from tilesparsity_b200 import TWLayer, _lib, tiles
    K, N = 1 << 19, 1 << 18
    col = np.ones(N, bool)
    col[5::1000] = False
    n_tiles = len(tiles.tile_bounds_from_col_mask(col, 128)) - 1
    rows = [np.arange(8, dtype=np.int32)] * n_tiles
    layer = TWLayer(tiles.tiles_from_lists(K, N, 128, rows, col), torch.float16, "cuda")
    assert layer.stats()["n_tiles"] == n_tiles
    rows = [np.arange(K, dtype=np.int32)] + rows[1:]
    with pytest.raises(_lib.TileSparseError):
        layer.retile(tiles.tiles_from_lists(K, N, 128, rows, col))
    x = torch.zeros((K, 8), dtype=torch.float16, device="cuda")
    for out in (None, torch.zeros((N, 8), dtype=torch.float16, device="cuda")):
        with pytest.raises(_lib.TileSparseError):
            layer.masked_gemm(x, out=out)
    assert _lib.lib.ts_layer_zero_pruned(layer._h, 8, out.data_ptr(), 8, None) == 1       # TS_ERR_INVALID
    torch.cuda.synchronize()
    assert layer.stats()["n_tiles"] == 0
    layer.close()


@pytest.mark.parametrize("n_streams", [2, 4, 6])          # 6: more than a layer has scratch memory for at a time
def test_split_k_on_several_streams(n_streams):
    """A layer whose long tiles are cut into ranges, used on several streams at once with other activations each, a
    captured graph among them: every product is its own (the ranges' partial sums do not meet)."""
    from tilesparsity_b200 import _lib
    K, N, M = 8192, 256, 64
    layer, W = _layer(K, N, 6000, torch.float16, 21)
    parts = (C.c_int32 * 2)()
    counts = (C.c_int32 * 2)(6000, 6000), (C.c_int32 * 2)(128, 128)
    assert _lib.lib.ts_plan_split(2, *counts, K, M, 148, parts) == 0 and max(parts) > 1
    xs = [torch.randn((K, M), device="cuda", generator=torch.Generator("cuda").manual_seed(i)).half() for i in range(n_streams)]
    refs = [layer.masked_gemm(x) for x in xs]
    Wm = _dense(W, layer, torch.float16)
    assert all(_rel(r, Wm.t() @ x.double()) <= TOL[torch.float16] for r, x in zip(refs, xs))
    outs = [[torch.zeros_like(refs[0]) for _ in range(50)] for _ in xs]
    held = torch.zeros_like(refs[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        layer.masked_gemm(xs[0], out=held)
    torch.cuda.synchronize()
    errors = []

    def work(i):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                for o in outs[i]:
                    layer.masked_gemm(xs[i], out=o)
                    if i == 0:
                        graph.replay()
            s.synchronize()
        except Exception as e:      # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(n_streams)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors
    assert all(torch.equal(o, r) for os, r in zip(outs, refs) for o in os)
    assert torch.equal(held, refs[0])
    layer.check()
    layer.close()


@pytest.mark.parametrize("K,N,keep,M,col_keep", [(8192, 4096, 4096, 4104, None),      # lists and plan of more than 256 KiB: copied piece by piece
                                                 (8192, 2048, 4000, 72, 0.9)])        # the lists only, with pruned columns
def test_large_lists_and_plans(K, N, keep, M, col_keep):
    layer, W = _layer(K, N, keep, torch.float16, 31, col_keep)
    x = torch.randn((K, M), device="cuda", generator=torch.Generator("cuda").manual_seed(M)).half()
    for _ in range(2):
        assert _rel(layer.masked_gemm(x), _dense(W, layer, torch.float16).t() @ x.double()) <= TOL[torch.float16]
        layer.retile(layer.tiles)
        layer.pack(W)
    layer.check()
    layer.close()


def test_large_plans_are_given_back():
    """Four plans of 9 MB each: re-tiling the layer gives all but a few megabytes of them back to the device."""
    layer, W = _layer(4096, 4096, 1024, torch.float16, 41)
    x = torch.zeros((4096, 16384), dtype=torch.float16, device="cuda")
    out = torch.zeros((4096, 16384), dtype=torch.float16, device="cuda")
    for i in range(4):
        layer.masked_gemm(x[:, :16384 - 8 * i], out=out[:, :16384 - 8 * i])
    gc.collect()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    layer.retile(layer.tiles)
    assert torch.cuda.mem_get_info()[0] - before >= 4 * 9e6 - (8 << 20) - (4 << 20)      # (4 MB: page granularity)
    layer.close()


def test_plans_of_graphs_stay_until_they_are_asked_for():
    """30 shapes of the reference-signature call, a graph each (plans of 20 MB): all plans stay, for a graph may hold
    them, until the program asks for their memory."""
    from tilesparsity_b200 import stream_gemm
    stream_gemm.trim_plans()
    M, N, K, G = 12800, 4096, 2048, 128
    flat_a, flat_c = (torch.zeros((n * M,), dtype=torch.float16, device="cuda") for n in (K, N))
    B = torch.zeros((N, K), dtype=torch.float16, device="cuda")
    lists = torch.zeros((K,), dtype=torch.int32, device="cuda")
    n = N // G

    def call(m):
        return stream_gemm.prepare_stream_gemm_nn(m, N, K, 1.0, flat_a[:K * m].view(K, m), B, 0.0, flat_c[:N * m].view(N, m), n, [G] * n, [K] * n,
                                                  [lists[:G]] * n, [lists] * n, [K * G * t for t in range(n)], [m * G * t for t in range(n)])

    def in_use():      # what is allocated on the device behind torch's back
        free, total = torch.cuda.mem_get_info()
        return total - free - torch.cuda.memory_reserved()

    graphs = []
    gc.collect()
    start = in_use()
    for i in range(30):
        c = call(M - 8 * i)
        c()
        torch.cuda.synchronize()
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            c()
    for g in graphs:
        g.replay()
    torch.cuda.synchronize()
    held = in_use() - start
    assert held > 30 * 10e6
    graphs.clear()
    g = None
    stream_gemm.trim_plans()
    assert in_use() - start < held * 0.1
    call(M)()
    torch.cuda.synchronize()


def test_a_graph_outlives_many_batch_sizes():
    """A captured product, then more batch sizes than a layer keeps plans for: the graph's plan stays, and its replay is
    the product of what its input holds by then."""
    layer, W = _layer(512, 384, 100, torch.float16, 51)
    x, out = torch.randn((512, 520), device="cuda").half(), torch.zeros((384, 520), dtype=torch.float16, device="cuda")
    layer.masked_gemm(x, out=out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        layer.masked_gemm(x, out=out)
    for i in range(1, 40):
        layer.masked_gemm(torch.randn((512, 8 * i), device="cuda").half())
    x.copy_(torch.randn((512, 520), device="cuda").half())
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert _rel(out, _dense(W, layer, torch.float16).t() @ x.double()) <= TOL[torch.float16]
    layer.check()
    del graph
    layer.close()


def test_threads_that_plan_and_ask():
    """Products of new batch sizes on one thread while others ask for schedules of others: one of them at a time."""
    layer, W = _layer(256, 512, 100, torch.float16, 61)
    Wm = _dense(W, layer, torch.float16)
    xs = [torch.randn((256, 8 * m), device="cuda").half() for m in range(1, 40)]
    torch.cuda.synchronize()
    errors, outs = [], {}

    def ask(first):
        try:
            for m in range(first, 400, 3):
                assert layer.schedule_stats(8 * m)["n_units"] > 0
        except Exception as e:      # reported by the main thread
            errors.append(e)

    def run():
        try:
            for i, x in enumerate(xs):
                outs[i] = layer.masked_gemm(x)
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=ask, args=(i,)) for i in (1, 2, 3)] + [threading.Thread(target=run)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors
    for i, x in enumerate(xs):
        assert _rel(outs[i], Wm.t() @ x.double()) <= TOL[torch.float16]
    layer.close()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("all_written", [True, False])
@pytest.mark.parametrize("K,N,M", [(64, 5, 8), (300, 130, 264), (1000, 64, 520)])
def test_residual_gemm(K, N, M, all_written, dtype):
    """ts_residual_gemm against float64, element by element.  fp16 adds up four products at a time in half precision (at
    most three roundings of 2^-11 of their magnitudes, and the products' own), bf16 in fp32; the output rounds once."""
    from tilesparsity_b200 import _lib
    g = torch.Generator("cuda").manual_seed(K + N + M)
    mask = torch.rand((K, N), device="cuda", generator=g) < 0.05
    mask[:, 1] = False                                   # a column without elements
    W = torch.randn((K, N), device="cuda", generator=g).to(dtype) * mask
    x = torch.randn((K, M), device="cuda", generator=g).to(dtype)
    Ct = torch.randn((N, M), device="cuda", generator=g).to(dtype)
    written = torch.ones(N, dtype=torch.uint8, device="cuda")
    if not all_written:
        written[::3] = 0
    at = mask.t().nonzero()                              # by column, rows ascending
    ptr = torch.zeros(N + 1, dtype=torch.int32, device="cuda")
    ptr[1:] = mask.sum(0).cumsum(0)
    rows, val = at[:, 1].int().contiguous(), W.t()[mask.t()].contiguous()
    alpha = -1.5
    base = Ct.double() * written[:, None]
    ref = base + alpha * (W.double().t() @ x.double())
    size = base.abs() + 1.5 * (W.double().abs().t() @ x.double().abs())
    p = lambda t: t.data_ptr()
    assert _lib.lib.ts_residual_gemm(0 if dtype == torch.float16 else 1, M, N, p(ptr), p(rows), p(val), None if all_written else p(written), p(x),
                                     x.stride(0), p(Ct), Ct.stride(0), alpha, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    unit = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    bound = unit * ref.abs() + (4 * 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -18) * size + 2.0 ** -20
    assert bool(((Ct.double() - ref).abs() <= bound).all())
