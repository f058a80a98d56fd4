"""Tensor-core kernels at the ends of the range of stationary tiles, against the fp64 closed form.
Few: the streamed tiles of one are shared by a cluster of CTAs (the cluster sizes that the rule takes,
read from captured launches; shares without a tile or without a visible key; both tile widths and types).
Many: two CTAs per SM, and persistent CTAs."""
import importlib
import re

import pytest
import torch

import attention_oracle as orc
from _util import captured_kernels

pytestmark = pytest.mark.gpu
tcapi = importlib.import_module("610sample_b200.torch_capi")
capi = importlib.import_module("610sample_b200.capi")

OUTPUTS = ("O", "dQ", "dK", "dV", "g_dO", "g_Q", "g_K", "g_V")
# Operands P and dS and the results are rounded to the type, each to u = 2^-9 (bf16) or 2^-12 (f16) of itself: 4 u of
# an output's norm, 8 u of its largest value for a single element.  A lost tile of 64 keys in 4096 is 12 % of the norm.
UNIT = {torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -12}


def _three_operations(g, window, chunk, mask):
    O, L = tcapi.forward(g["Q"], g["K"], g["V"], window, chunk, mask)
    b = tcapi.backward(g["dO"], g["Q"], g["K"], g["V"], O, L, window, chunk, mask)
    h = tcapi.double_backward(g["g_dQ"], g["g_dK"], g["g_dV"], g["dO"], g["Q"], g["K"], g["V"], O, L, window, chunk, mask)
    return L, (O,) + tuple(b) + tuple(h)


def _check_against_the_oracle(B, H, N_q, N_kv, D, window, chunk, mask, dtype):
    inp = orc.make_inputs(B, H, N_q, N_kv, D, seed=N_q + N_kv, dtype=dtype)
    ref = orc.closed_form_all(*(inp[n] for n in orc.INPUT_NAMES), window_size=window, chunk_id=chunk, mask_mode=mask, device="cuda")
    g = {n: t.cuda() for n, t in inp.items()}
    L, first = _three_operations(g, window, chunk, mask)
    _, second = _three_operations(g, window, chunk, mask)
    assert torch.allclose(L.cpu().double(), ref["L"].double(), rtol=1e-5, atol=1e-4)
    for got, again, n in zip(first, second, OUTPUTS):
        assert torch.equal(got, again), n
        r = ref[n].double()
        diff = got.double().cpu() - r
        assert float(diff.norm()) <= 4 * UNIT[dtype] * float(r.norm()), n
        assert float(diff.abs().max()) <= 8 * UNIT[dtype] * float(r.abs().max()), n
    assert capi.device_status() == 0
    return g


def _clusters(g, window, chunk, mask):
    """{kernel: CTAs per cluster} of the three operations, from a captured graph."""
    drv = pytest.importorskip("cuda.bindings.driver")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        keep = _three_operations(g, window, chunk, mask)
    raw = drv.CUgraph(graph.raw_cuda_graph())
    _, _, n = drv.cuGraphGetNodes(raw, 0)
    _, nodes, _ = drv.cuGraphGetNodes(raw, n)
    found = {}
    for node in nodes:
        if drv.cuGraphNodeGetType(node)[1] != drv.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        p = drv.cuGraphKernelNodeGetParams(node)[1]
        name = (drv.cuFuncGetName(p.func) if int(p.func) else drv.cuKernelGetName(p.kern))[1].decode()
        attr = drv.cuGraphKernelNodeGetAttribute(node, drv.CUkernelNodeAttrID.CU_LAUNCH_ATTRIBUTE_CLUSTER_DIMENSION)[1]
        for part, kernel in (("fwd_kernel", "O"), ("fb_kernelILi2E", "dQ"), ("fb_kernelILi3E", "dK"), ("hvp_row_kernelILi0E", "g_dO"),
                             ("hvp_row_kernelILi1E", "g_Q"), ("hvp_col_kernel", "g_K")):
            if part in name:
                found[kernel] = max(1, attr.clusterDim.x)
    del keep
    return found


# (heads, queries, keys, D, window, chunk, mask): kernels whose tiles are shared there
SPLIT = [
    ((1, 128, 4096, 64, 4096, 0, 1), "O dQ g_dO g_Q"),            # one tile of queries against 64 of keys
    ((1, 100, 1999, 128, 1999, 30, 0), "O dQ g_dO g_Q"),          # ragged on both axes
    ((1, 128, 2048, 64, 700, 15, 0), "O dQ g_dO g_Q"),            # window: shares that half of the rows do not see
    ((1, 128, 2048, 128, 1500, 15, 0), "O dQ g_dO g_Q"),
    ((1, 2048, 2048, 64, 2048, 0, 0), "O g_dO dK"),               # causal: tiles of 2 to 32, shares without any
    ((1, 2048, 2048, 128, 2048, 0, 0), "O g_dO dK"),
    ((1, 4096, 128, 64, 4096, 0, 1), "dK g_K"),                   # the key side is the short one
    ((1, 4000, 100, 128, 4096, 0, 1), "dK g_K"),
    ((7, 4096, 128, 128, 4096, 0, 1), "dK g_K"),
    ((8, 4096, 128, 64, 4096, 0, 1), "dK g_K"),
    ((11, 4096, 128, 64, 4096, 0, 1), "dK g_K"),
    ((14, 4000, 100, 80, 4096, 0, 1), "dK g_K"),
    ((16, 4096, 128, 64, 4096, 0, 1), "dK g_K"),
    ((7, 128, 4096, 64, 4096, 0, 1), "O dQ g_dO g_Q"),
    ((8, 100, 4000, 80, 4096, 0, 1), "O dQ g_dO g_Q"),
    ((9, 128, 4096, 128, 4096, 0, 1), "O dQ g_dO g_Q"),
    ((12, 128, 4096, 64, 4096, 0, 1), "O dQ g_dO g_Q"),
    ((20, 128, 4096, 128, 4096, 0, 1), "O g_dO g_Q"),
    ((24, 128, 4096, 64, 4096, 0, 1), "O g_dO"),
    ((30, 100, 4000, 96, 4096, 0, 1), "O g_dO"),
    ((36, 128, 4096, 64, 4096, 0, 1), "O g_dO"),
    ((60, 128, 4096, 128, 4096, 0, 1), "O g_dO"),
]
SIZES = {}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape,kernels", SPLIT)
def test_shared_tiles_match_the_oracle(shape, kernels, dtype):
    H, N_q, N_kv, D, window, chunk, mask = shape
    g = _check_against_the_oracle(1, H, N_q, N_kv, D, window, chunk, mask, dtype)
    found = _clusters(g, window, chunk, mask)
    assert len(found) == 6
    for k in kernels.split():
        assert found[k] > 1, (k, found)
    for k, c in found.items():
        SIZES.setdefault((k, D > 64), set()).add(c)


def test_shared_tiles_cover_the_range_of_sizes():
    """What the cases above have launched: at least four sizes of every kernel, pairs and eights among
    them, in either tile width."""
    if len(SIZES) < 12:
        pytest.skip("needs the cases above")
    for k in ("O", "dQ", "dK", "g_dO", "g_Q", "g_K"):
        narrow, wide = SIZES[k, False] - {1}, SIZES[k, True] - {1}
        assert 8 in narrow and 8 in wide and len(narrow | wide) >= 4 and min(narrow | wide) <= 3, (k, narrow, wide)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,N_q,N_kv,D,window,chunk,mask", [
    (1, 2, 257, 900, 80, 300, 3, 0),         # window: the range of a tile starts inside a 64-row tile
    (2, 3, 130, 1000, 96, 1000, 0, 0),       # most keys in front of the sequence
    (1, 1, 64, 190, 64, 190, 9, 0),          # three tiles
    (1, 1, 1500, 130, 128, 1500, 0, 1),      # the key side is the short one
    (1, 5, 640, 640, 64, 640, 0, 0),         # causal: tiles of 2 to 10
    (3, 16, 300, 1300, 128, 1000, 2, 0),     # 144 tiles: no cluster
    (1, 1, 70, 600, 16, 40, 0, 0),           # keys without a visible query
    (8, 40, 129, 129, 64, 129, 0, 0),        # two CTAs per SM, one row in every second tile
    (4, 50, 300, 520, 48, 200, 1, 0),        # the same with padding, a window and keys nobody sees
    (6, 50, 60, 190, 64, 190, 0, 1),         # one tile per head
    (5, 40, 200, 200, 128, 200, 0, 0),       # two forward CTAs per SM, Q in shared memory
    (4, 40, 190, 500, 80, 130, 1, 0),        # the same with padding and a window
    (2, 200, 130, 70, 64, 20, 0, 0),         # persistent CTAs: items of one or two tiles
    (2, 80, 300, 900, 128, 100, 0, 0),       # the same, and items without a tile in between
])
def test_few_and_many_tiles_match_the_oracle(B, H, N_q, N_kv, D, window, chunk, mask, dtype):
    _check_against_the_oracle(B, H, N_q, N_kv, D, window, chunk, mask, dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,N,D", [(2, 700, 64), (2, 700, 128), (120, 513, 64), (100, 385, 128)])
def test_forward_when_scores_grow_along_the_keys(H, N, D, dtype):
    """Keys that grow with their position make the reference exponent of most rows too low again and
    again (score maxima move by some 40 log2 units), in every variant of the forward."""
    inp = orc.make_inputs(1, H, N, N, D, seed=H + D, dtype=torch.float32)
    K = (inp["K"] * torch.linspace(0.1, 10.0, N).view(1, 1, N, 1)).to(dtype)
    Q, V = inp["Q"].to(dtype), inp["V"].to(dtype)
    for mask in (0, 1):
        O, L = tcapi.forward(Q.cuda(), K.cuda(), V.cuda(), N, 0, mask)
        S = torch.einsum("bhid,bhjd->bhij", Q.cuda().double(), K.cuda().double()) / D ** 0.5
        if mask == 0:
            S = S.masked_fill(torch.ones(N, N, device="cuda").triu(1).bool(), float("-inf"))
        want_L = torch.logsumexp(S, -1)
        want_O = torch.softmax(S, -1) @ V.cuda().double()
        # L: fp32 sums; O: P rounded to the type (relative 2^-9 or 2^-12 of a convex combination of V) and the result
        assert torch.allclose(L.double(), want_L, rtol=1e-5, atol=1e-4), mask
        tol = {torch.bfloat16: 2 ** -7, torch.float16: 2 ** -10}[dtype]
        assert float((O.double() - want_O).abs().max()) <= tol * float(V.double().abs().max()), mask


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,N,D", [(8, 768, 64), (160, 512, 64), (100, 384, 128)])      # one and two CTAs per SM
def test_tiles_done_again_keep_their_second_result(H, N, D, dtype):
    """Every tile of 64 keys is far above the one before it, so that the forward does every tile of a
    row twice: what stays must be the second P, bit for bit the same in every run."""
    inp = orc.make_inputs(1, H, N, N, D, seed=7, dtype=torch.float32)
    Q = torch.full((1, H, N, D), 0.25) + 0.01 * inp["Q"]
    K = ((torch.arange(N) // 64).view(1, 1, N, 1) * (80.0 / D ** 0.5) + 0.01 * inp["K"]).to(dtype)      # 28 log2 units a tile
    Q, V = Q.to(dtype), inp["V"].to(dtype)
    q, k, v = Q.cuda(), K.cuda(), V.cuda()
    first, L = tcapi.forward(q, k, v, N, 0, 1)
    S = torch.einsum("bhid,bhjd->bhij", q.double(), k.double()) / D ** 0.5
    want = torch.softmax(S, -1) @ v.double()
    assert torch.allclose(L.double(), torch.logsumexp(S, -1), rtol=1e-5, atol=1e-4)
    tol = {torch.bfloat16: 2 ** -7, torch.float16: 2 ** -10}[dtype]      # as above
    assert float((first.double() - want).abs().max()) <= tol * float(v.double().abs().max())
    for _ in range(50):
        assert torch.equal(tcapi.forward(q, k, v, N, 0, 1)[0], first)


@pytest.mark.parametrize("dtype,bound", [(torch.bfloat16, 2.15e-3), (torch.float16, 2.6e-4)])
@pytest.mark.parametrize("B,H,N,D", [(4, 16, 1024, 128), (4, 16, 4096, 128), (8, 12, 1024, 64), (8, 12, 300, 64), (1, 4, 1024, 64)])
def test_forward_of_peaked_rows_is_as_exact_as_its_type(B, H, N, D, dtype, bound):
    """Scores of standard deviation 4: a row is little else than its largest P, which has to be close to
    one to be exact in half precision.  Relative error of O: the rounding of the result is 1.66e-3 (bf16;
    an eighth of that in f16), a reference exponent that follows the maximum adds up to 2.05e-3 in all, one
    that lags behind it as far as the type allows 2.3e-3 (f16: 2.45e-4 and 2.75e-4)."""
    inp = orc.make_inputs(B, H, N, N, D, seed=N, dtype=torch.float32)
    Q, K, V = ((inp[n] * a).to(dtype).cuda() for n, a in (("Q", 2.0), ("K", 2.0), ("V", 1.0)))
    O, _ = tcapi.forward(Q, K, V, N, 0)
    err = norm = 0.0
    for b, h in ((0, 0), (B - 1, H - 1), (0, H // 2)):
        S = (Q[b, h].double() @ K[b, h].double().T / D ** 0.5).masked_fill(torch.ones(N, N, device="cuda").triu(1).bool(), float("-inf"))
        want = torch.softmax(S, -1) @ V[b, h].double()
        err += float((O[b, h].double() - want).pow(2).sum())
        norm += float(want.pow(2).sum())
    assert (err / norm) ** 0.5 <= bound


def test_split_rows_without_a_sum_are_those_of_the_unsplit_kernel():
    """One key with an infinite element: rows whose score with it is +inf have no sum (L = -inf) and get
    zeros, split or not; rows whose score is -inf do not see the key."""
    N, D = 2048, 64
    inp = orc.make_inputs(1, 1, 128, N, D, seed=9, dtype=torch.bfloat16)
    Q, K, V = (inp[n].cuda() for n in ("Q", "K", "V"))
    K[0, 0, 70, 3] = float("inf")
    many = [t.expand(1, 160, -1, -1).contiguous() for t in (Q, K, V)]
    for q, k, v in ((Q, K, V), many):
        O, L = tcapi.forward(q, k, v, N, 15, 1)
        lost = Q[0, 0, :, 3] > 0
        assert bool(torch.isneginf(L[0, 0, lost]).all()) and float(O[0, 0, lost].float().abs().max()) == 0.0
        S = (Q[0, 0].double() @ K[0, 0].double().T / D ** 0.5)[~lost]
        want = torch.softmax(S, -1) @ V[0, 0].double()
        assert float((O[0, 0, ~lost].double() - want).abs().max()) <= 2 ** -7 * float(V.double().abs().max())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,D", [(10, 64), (60, 64), (10, 80), (10, 112), (10, 128)])      # one CTA per SM, two (60 heads)
def test_first_backward_in_one_grid_and_in_two_gives_the_same_bits(H, D, dtype):
    """1000 queries at the start of the sequence against 3048 keys, 2048 of them in front of it: no window from 1000 on
    hides a key, but a wide one makes the bound of the streamed tiles 48 instead of 19, so dQ and dK/dV
    get a launch each."""
    inp = orc.make_inputs(1, H, 1000, 3048, D, seed=H + D, dtype=dtype)
    g = {n: t.cuda() for n, t in inp.items()}
    results = []
    for window, launches in ((1000, ["pair"]), (8192, ["tile", "tile"])):
        O, L = tcapi.forward(g["Q"], g["K"], g["V"], window, 0, 0)
        call = lambda: tcapi.backward(g["dO"], g["Q"], g["K"], g["V"], O, L, window, 0, 0)
        assert [n.split("_kernel")[0][-4:] for n, c in captured_kernels(call) if "fb_kernel" in n] == launches
        results.append((O, L) + tuple(call()))
    assert float(results[0][3][:, :, 2048:].float().norm()) > 0
    for one, two, name in zip(*results, ("O", "L", "dQ", "dK", "dV")):
        assert torch.equal(one, two), name


def _backward_forms(call):
    """[two CTAs per SM] of each launch of the first backward's tiles (both kinds of a pair have the same form)."""
    kernels = [n for n, _ in captured_kernels(call) if "fb_kernel" in n]
    forms = [f for n in kernels for f in re.findall(r"fb_kernelILi\d+ELi64E.*?Lb[01]ELb([01])E", n)[:1]]
    assert len(forms) == len(kernels), kernels
    return [f == "1" for f in forms]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape,forms", [
    ((24, 1000, 1000, 64, 1000, 0, 0), [True]),         # causal, ragged: 192 tiles of either side
    ((32, 700, 1500, 48, 333, 2, 0), [True]),           # both edges of a window inside the tiles
    ((48, 500, 450, 64, 500, 0, 1), [True]),            # no mask: equal CTAs of short streams, the ends of both axes
    ((80, 250, 250, 64, 20, 0, 0), [True]),             # a narrow window: most scores of every tile masked
    ((10, 2000, 2000, 64, 2000, 0, 0), [False]),        # few tiles, long streams: the longest CTA would be the bound
    ((28, 778, 1139, 64, 778, 0, 1), [True]),           # no mask: more than three rounds of CTAs, both kinds together
    ((24, 1060, 1060, 64, 1060, 0, 1), [False]),        # no mask: three rounds
    ((16, 1600, 2200, 64, 1600, 0, 1), [True, True]),   # streams of more than 33 tiles: a launch for each kind
    ((20, 128, 1374, 64, 1246, 0, 0), [False]),         # 220 tiles of keys, 180 of them in front of the sequence
    ((24, 187, 1440, 48, 1253, 5, 0), [False, True]),   # fewer tiles of queries than SMs: the keys' kind decides by itself
])
def test_first_backward_with_two_ctas_per_sm(shape, forms, dtype):
    H, N_q, N_kv, D, window, chunk, mask = shape
    g = _check_against_the_oracle(1, *shape, dtype)
    O, L = tcapi.forward(g["Q"], g["K"], g["V"], window, chunk, mask)
    got = _backward_forms(lambda: tcapi.backward(g["dO"], g["Q"], g["K"], g["V"], O, L, window, chunk, mask))
    assert sorted(got) == forms


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_first_backward_with_one_and_two_ctas_per_sm_gives_the_same_bits(dtype):
    """24 heads have two CTAs per SM, the first 10 of them by themselves one; neither form shares a tile over a cluster."""
    N = 1000
    g = {n: t.cuda() for n, t in orc.make_inputs(1, 24, N, N, 64, seed=24, dtype=dtype).items()}
    args = [g["dO"], g["Q"], g["K"], g["V"], *tcapi.forward(g["Q"], g["K"], g["V"], N, 0, 0)]
    few = [t[:, :10].contiguous() for t in args]
    calls = [lambda a=a: tcapi.backward(*a, N, 0, 0) for a in (args, few)]
    assert [_backward_forms(c) for c in calls] == [[True], [False]]
    for two, one, name in zip(calls[0](), calls[1](), ("dQ", "dK", "dV")):
        assert torch.equal(two[:, :10], one), name


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape,two", [
    ((96, 250, 250, 96, 250, 0, 0), True),          # short streams of unequal length
    ((24, 1500, 1500, 64, 1500, 0, 0), False),
    ((20, 1000, 1100, 64, 1000, 0, 1), True),       # no mask: two rounds of 148 CTAs, short streams
    ((22, 900, 3100, 80, 2200, 3, 0), False),       # a window: two rounds, long streams
    ((148, 120, 200, 64, 200, 0, 1), False),        # one round
])
def test_forward_with_two_ctas_per_sm(shape, two, dtype):
    H, N_q, N_kv, D, window, chunk, mask = shape
    g = _check_against_the_oracle(1, *shape, dtype)
    kernels = [n for n, _ in captured_kernels(lambda: tcapi.forward(g["Q"], g["K"], g["V"], window, chunk, mask)) if "fwd_kernel" in n]
    forms = [f for n in kernels for f in re.findall(r"fwd_kernelILi\d+E.*?Lb[01]ELi([12])E", n)]      # groups of math warps of a CTA
    assert forms == ["1" if two else "2"], kernels
