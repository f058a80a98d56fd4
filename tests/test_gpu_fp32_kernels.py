"""fp32 kernels at the edges of their tiles and at every size of the cluster split: 32 stationary and
64 streamed rows per tile, 1 / 2 / 4 / 8 CTAs per stationary tile, both tile widths, head dimensions
with and without the swizzled layout."""
import importlib

import pytest
import torch

import attention_oracle as orc
from _util import captured_kernels

pytestmark = pytest.mark.gpu
tcapi = importlib.import_module("610sample_b200.torch_capi")


@pytest.mark.parametrize("B,H,N_q,N_kv,D,window,chunk,mask", [
    (1, 1, 32, 64, 64, 64, 0, 1),        # exactly one tile
    (1, 1, 33, 65, 48, 40, 1, 0),        # one row more on both axes; pitch with padding
    (1, 2, 31, 129, 128, 1000, 0, 0),    # split 2, last part nearly empty
    (1, 1, 95, 250, 80, 250, 2, 0),      # split 4
    (1, 2, 64, 520, 64, 520, 3, 0),      # split 8; keys in front of the sequence in no window
    (2, 1, 64, 520, 16, 70, 9, 0),       # a window shorter than the keys: parts without a visible key
    (2, 8, 600, 600, 64, 600, 0, 0),     # no split
    (1, 3, 40, 1, 96, 1, 0, 1),          # one key
])
def test_fp32_kernels_match_the_oracle(B, H, N_q, N_kv, D, window, chunk, mask):
    inp = orc.make_inputs(B, H, N_q, N_kv, D, seed=N_q + D, dtype=torch.float32)
    ref = orc.closed_form_all(*(inp[n] for n in orc.INPUT_NAMES), window_size=window, chunk_id=chunk, mask_mode=mask)
    g = {n: t.cuda() for n, t in inp.items()}
    runs = []
    for _ in range(2):
        O, L = tcapi.forward(g["Q"], g["K"], g["V"], window, chunk, mask)
        b = tcapi.backward(g["dO"], g["Q"], g["K"], g["V"], O, L, window, chunk, mask)
        h = tcapi.double_backward(g["g_dQ"], g["g_dK"], g["g_dV"], g["dO"], g["Q"], g["K"], g["V"], O, L, window, chunk, mask)
        runs.append((O,) + tuple(b) + tuple(h))
    for got, again, n in zip(*runs, ("O", "dQ", "dK", "dV", "g_dO", "g_Q", "g_K", "g_V")):
        assert torch.equal(got, again), n
        r = ref[n].double()
        # the family's stated tolerance: 1e-4 of the largest value (fp32 sums of at most N * D terms)
        assert float((got.double().cpu() - r).abs().max()) <= 1e-4 * max(1.0, float(r.abs().max())), n


@pytest.mark.parametrize("B,H,N,D,impl,dtype", [(1, 4, 256, 64, 0, torch.float32), (2, 16, 500, 80, 0, torch.float32),
                                                (1, 2, 200, 128, 1, torch.bfloat16)])
def test_a_query_that_is_not_a_number_gives_a_row_that_is_not(B, H, N, D, impl, dtype):
    inp = orc.make_inputs(B, H, N, N, D, seed=5, dtype=dtype)
    Q, K, V = (inp[n].cuda() for n in ("Q", "K", "V"))
    want, _ = tcapi.forward(Q, K, V, N, 0, 0, impl)
    Q[:, 0, 7, 3] = float("nan")
    O, _ = tcapi.forward(Q, K, V, N, 0, 0, impl)
    assert bool(torch.isnan(O[:, 0, 7]).all())
    O[:, 0, 7] = want[:, 0, 7]
    assert torch.equal(O, want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,N_q,N_kv,D", [(1, 4, 300, 400, 64), (4, 24, 256, 320, 80)])      # a cluster per tile, none
def test_half_inputs_give_the_rounded_exact_result(B, H, N_q, N_kv, D, dtype):
    """The arithmetic is fp32, so the double backward is the exact one but for the rounding of its results
    (g_dK has a mean, so that dot2 O is as large as the sum it is taken from)."""
    inp = orc.make_inputs(B, H, N_q, N_kv, D, seed=3, dtype=torch.float32)
    inp["g_dK"] = inp["g_dK"] + 1.0
    inp = {n: t.to(dtype) for n, t in inp.items()}
    ref = orc.closed_form_all(*(inp[n] for n in orc.INPUT_NAMES), window_size=N_kv, chunk_id=2, device="cuda")
    g = {n: t.cuda() for n, t in inp.items()}
    O, L = tcapi.forward(g["Q"], g["K"], g["V"], N_kv, 2, 0, 1)
    h = tcapi.double_backward(g["g_dQ"], g["g_dK"], g["g_dV"], g["dO"], g["Q"], g["K"], g["V"], O, L, N_kv, 2, 0, 1)
    # sums of 400 terms in fp32 are off by some 1e-6 of the sum's terms, a 2^10-th (f16) of the step from one result to the
    # next: few results are rounded to the other side
    for got, n in zip(h, ("g_dO", "g_Q", "g_K", "g_V")):
        assert float((got.cpu() != ref[n].to(dtype)).float().mean()) <= 0.02, n


def _forms(g, window, chunk, mask):
    """{kernel: CTAs per cluster} of the three operations, "dK+dQ" where two of them are one grid."""
    def call():
        O, L = tcapi.forward(g["Q"], g["K"], g["V"], window, chunk, mask)
        b = tcapi.backward(g["dO"], g["Q"], g["K"], g["V"], O, L, window, chunk, mask)
        return O, b, tcapi.double_backward(g["g_dQ"], g["g_dK"], g["g_dV"], g["dO"], g["Q"], g["K"], g["V"], O, L, window, chunk, mask)
    kinds = {"kernelILi0E": "O", "kernelILi1E": "dQ", "kernelILi2E": "dK", "kernelILi3E": "g_dO", "kernelILi4E": "g_Q", "kernelILi5E": "g_K",
             "pair_kernelILi2ELi1E": "dK+dQ", "pair_kernelILi5ELi4E": "g_K+g_Q"}
    found = {}
    for name, cluster in captured_kernels(call):
        for part in sorted(kinds, key=len, reverse=True):
            if "attn_simt_" + part in name:
                found[kinds[part]] = cluster
                break
    return found


def _parsed(forms):
    words = forms.split()
    return {k: int(c) for k, c in zip(words[::2], words[1::2])}


# (B, H, N_q, N_kv, D, window, chunk, mask) and the forms that the rule takes there
FORMS = [
    ((2, 5, 479, 479, 64, 479, 0, 0), "O 2 dQ 2 dK 2 g_dO 4 g_Q 4 g_K 2"),            # 150 tiles of up to 8: parts without a tile
    ((4, 1, 383, 383, 48, 383, 0, 0), "O 4 dQ 4 dK 4 g_dO 4 g_Q 4 g_K 4"),
    ((1, 1, 700, 700, 64, 700, 0, 0), "O 8 dQ 8 dK 8 g_dO 8 g_Q 8 g_K 8"),
    ((1, 3, 150, 150, 128, 150, 0, 0), "O 4 g_dO 4 dK+dQ 4 g_K+g_Q 4"),               # three streamed tiles for a cluster of four
    ((2, 7, 160, 293, 80, 293, 1, 0), "O 2 g_dO 2 dK+dQ 1 g_Q 2 g_K 1"),              # 140 and 70 tiles: one side split
    ((2, 5, 160, 293, 80, 293, 1, 0), "O 4 dQ 2 dK 1 g_dO 4 g_Q 2 g_K 1"),
    ((1, 9, 1023, 65, 64, 1023, 0, 1), "O 1 dQ 1 dK 8 g_dO 1 g_Q 1 g_K 8"),           # 288 tiles of two, 27 of 16
    ((1, 10, 961, 33, 96, 40, 0, 0), "O 1 dQ 1 dK 2 g_dO 1 g_Q 1 g_K 2"),             # 310 tiles, most of which see nothing
    ((1, 1, 520, 520, 64, 520, 0, 0), "O 8 g_dO 8 dK+dQ 8 g_K+g_Q 8"),
    ((1, 1, 400, 400, 64, 400, 0, 0), "O 8 g_dO 8 dK+dQ 8 g_K+g_Q 8"),
    ((1, 1, 520, 520, 128, 520, 0, 0), "O 8 g_dO 8 dK+dQ 4 g_K+g_Q 4"),
    ((1, 1, 300, 300, 80, 300, 0, 0), "O 8 dQ 4 dK 8 g_dO 8 g_Q 4 g_K 8"),
    ((1, 1, 33, 500, 96, 500, 0, 1), "O 8 dQ 8 dK 1 g_dO 8 g_Q 8 g_K 1"),
    ((1, 1, 500, 33, 112, 500, 0, 1), "O 1 dQ 1 dK 8 g_dO 1 g_Q 1 g_K 8"),
    ((1, 1, 95, 250, 80, 250, 2, 0), "O 4 dQ 4 dK 2 g_dO 4 g_Q 4 g_K 2"),
    ((1, 4, 100, 100, 64, 100, 0, 0), "O 2 g_dO 2 dK+dQ 2 g_K+g_Q 2"),
    ((2, 2, 250, 250, 64, 250, 0, 0), "O 4 g_dO 4 dK+dQ 4 g_K+g_Q 4"),
    ((1, 1, 32, 64, 64, 64, 0, 1), "O 1 g_dO 1 dK+dQ 1 g_K+g_Q 1"),                   # one tile: one grid without a cluster
    ((2, 8, 600, 600, 64, 600, 0, 0), "O 1 dQ 1 dK 1 g_dO 1 g_Q 1 g_K 1"),            # 304 tiles: no split
    ((1, 1, 264, 586, 80, 586, 0, 0), "O 8 g_dO 8 dK+dQ 4 g_K+g_Q 8"),                # keys without a visible query
    ((2, 8, 300, 300, 80, 300, 0, 0), "O 1 g_dO 2 dK+dQ 1 g_Q 2 g_K 1"),
]


@pytest.mark.parametrize("shape,forms", FORMS)
def test_fp32_splits_match_the_oracle(shape, forms):
    B, H, N_q, N_kv, D, window, chunk, mask = shape
    test_fp32_kernels_match_the_oracle(*shape)
    g = {n: t.cuda() for n, t in orc.make_inputs(B, H, N_q, N_kv, D, seed=1, dtype=torch.float32).items()}
    assert _forms(g, window, chunk, mask) == _parsed(forms)


def test_fp32_forms_cover_every_kernel():
    """The cases above name each kernel without a split and in clusters of 2, 4 and 8, at D <= 64 and above, and both
    pairs as one grid."""
    seen = {}
    for shape, forms in FORMS:
        for kernel, c in _parsed(forms).items():
            for k in {kernel, *kernel.split("+")}:
                seen.setdefault((k, shape[4] > 64), set()).add(c)
    for wide in (False, True):
        for k in ("O", "dQ", "dK", "g_dO", "g_Q", "g_K"):
            assert seen[k, wide] == {1, 2, 4, 8}, (k, wide, seen[k, wide])
    assert seen["dK+dQ", False] == {1, 2, 4, 8} and seen["g_K+g_Q", False] == {1, 2, 4, 8}
    assert {1, 4} <= seen["dK+dQ", True] and {4, 8} <= seen["g_K+g_Q", True]
