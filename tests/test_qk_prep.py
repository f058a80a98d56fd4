"""The fused step before attention (RMS norm + rotary embedding + layout change): the oracle
restatement against the fixture made by the reference's own RMSNorm / apply_rotary_emb (CPU), and
the CUDA kernel and its differentiable wrapper against the oracle (GPU)."""
import importlib
import os
import sys

import pytest
import torch

import attention_oracle as orc
from _util import load_prep_golden

PKG_DIR = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "610sample_b200")


def test_oracle_matches_the_reference_fixture():
    m, x, w, want = load_prep_golden()
    fc = orc.rope_freqs_cis(m["d"], 128)
    got = orc.qk_norm_rope_oracle(x, w, fc, pos0=m["pos0"], eps=1e-6, norm_from=m["norm_from"])
    assert got.shape == want.shape == (1, m["H"], m["n_tok"], m["d"])
    assert torch.equal(got.float(), want)          # same operations in the same order: bit-exact


def test_oracle_without_weight_only_rotates():
    x = torch.randn(5, 2, 16)
    fc = orc.rope_freqs_cis(16, 8)
    y = orc.qk_norm_rope_oracle(x, None, fc)
    assert torch.allclose(y.norm(dim=-1)[0].T, x.norm(dim=-1), atol=1e-5)      # a rotation keeps the length
    assert torch.allclose(y[0, :, 0], x[0])                                    # position 0: identity


@pytest.fixture(scope="module")
def prep():
    if PKG_DIR not in sys.path:
        sys.path.insert(0, PKG_DIR)
    return importlib.import_module("qk_prep")


@pytest.mark.gpu
def test_kernel_matches_reference_fixture_and_oracle(prep):
    m, x, w, want = load_prep_golden()
    table = prep.rope_table(m["d"], 128, device="cuda")
    got = prep.qk_norm_rope(x.cuda(), w.cuda(), table, pos0=m["pos0"], eps=1e-6, norm_from=m["norm_from"])
    # fp32 arithmetic in a different summation order: at most one bf16 unit in the last place
    err = (got.float().cpu() - want).abs()
    assert float((err / want.abs().clamp_min(1e-3)).max()) <= 2 ** -7
    assert float((err > 0).float().mean()) < 0.02
    # the last three: a head count that is not a multiple of the four a lane group walks over, a
    # width of 8 lanes with a partly filled last CTA, and a head dimension (not a multiple of 8)
    # that takes the pairwise kernel
    for dtype, D, H, n in ((torch.float16, 128, 4, 300), (torch.float32, 80, 2, 77), (torch.bfloat16, 96, 16, 1024),
                           (torch.float16, 64, 5, 130), (torch.bfloat16, 16, 7, 33), (torch.bfloat16, 20, 3, 65)):
        xx = torch.randn(n, H, D).to(dtype)
        ww = (1 + 0.1 * torch.randn(D)).to(dtype)
        fc = orc.rope_freqs_cis(D, n + 9)
        ref = orc.qk_norm_rope_oracle(xx, ww, fc, pos0=9, norm_from=n // 3)
        out = prep.qk_norm_rope(xx.cuda(), ww.cuda(), prep.rope_table(D, n + 9, device="cuda"), pos0=9, norm_from=n // 3)
        tol = {torch.float16: 2 ** -9, torch.bfloat16: 2 ** -7, torch.float32: 1e-5}[dtype]      # a unit or two in the last place
        # a rotated element is a difference of two rounded products: its error scales with the inputs (O(1)), not with itself
        assert float(((out.float().cpu() - ref.float()).abs() / (1.0 + ref.float().abs())).max()) <= tol, dtype
        no_norm = prep.qk_norm_rope(xx.cuda(), None, prep.rope_table(D, n + 9, device="cuda"), pos0=9)
        ref2 = orc.qk_norm_rope_oracle(xx, None, fc, pos0=9)
        assert float((no_norm.float().cpu() - ref2.float()).abs().max()) <= tol * float(ref2.float().abs().max())


@pytest.mark.gpu
def test_kernel_full_tile_variant_matches_oracle(prep):
    """Shapes whose CTAs are all full and whose normalisation covers every token take the
    guard-free variant of the kernel; the same shapes with one token more take the guarded one,
    and the two agree bit for bit on the tokens they share."""
    for dtype, D, H, n in ((torch.bfloat16, 128, 8, 256), (torch.float16, 64, 4, 96), (torch.float32, 128, 4, 32),
                           (torch.bfloat16, 64, 12, 1024)):
        xx = torch.randn(n + 1, H, D).to(dtype)
        ww = (1 + 0.1 * torch.randn(D)).to(dtype)
        fc = orc.rope_freqs_cis(D, n + 4)
        table = prep.rope_table(D, n + 4, device="cuda")
        tol = {torch.float16: 2 ** -9, torch.bfloat16: 2 ** -7, torch.float32: 1e-5}[dtype]
        for weight in (ww, None):
            ref = orc.qk_norm_rope_oracle(xx[:n], weight, fc, pos0=3)
            wc = None if weight is None else weight.cuda()
            full = prep.qk_norm_rope(xx[:n].cuda(), wc, table, pos0=3)
            assert float(((full.float().cpu() - ref.float()).abs() / (1.0 + ref.float().abs())).max()) <= tol, (dtype, D)
            ragged = prep.qk_norm_rope(xx.cuda(), wc, table, pos0=3)
            assert torch.equal(ragged[:, :, :n], full), (dtype, D)


@pytest.mark.gpu
def test_wrapper_is_differentiable_to_second_order_and_feeds_attention(prep):
    """Gradients of the fused call equal those of the plain PyTorch formulas, first and second
    order, and its output goes straight into flash_attention_v7 (layout [1, H, n_tok, d])."""
    from attention import flash_attention_v7
    torch.manual_seed(5)
    n, H, D = 192, 2, 64
    x0 = torch.randn(n, H, D, device="cuda", dtype=torch.float32)
    w0 = (1 + 0.1 * torch.randn(D, device="cuda"))
    table = prep.rope_table(D, n, device="cuda")
    u = torch.randn(1, H, n, D, device="cuda")

    def second_order(fn):
        x = x0.clone().requires_grad_(True)
        w = w0.clone().requires_grad_(True)
        y = fn(x, w, table)
        gx, gw = torch.autograd.grad((y * u).sum() + (y * y).sum(), [x, w], create_graph=True)
        hx, hw = torch.autograd.grad(gx.pow(2).sum() + gw.pow(2).sum(), [x, w])
        return y, gx, gw, hx, hw

    got = second_order(prep.qk_norm_rope)
    want = second_order(prep.qk_norm_rope_torch)
    for a, b, name in zip(got, want, ("y", "gx", "gw", "hx", "hw")):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-4 * float(b.abs().max())), name

    xq = torch.randn(n, H, D, device="cuda").to(torch.bfloat16).requires_grad_(True)
    wq = torch.ones(D, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    Q = prep.qk_norm_rope(xq, wq, table)
    O = flash_attention_v7(Q, Q.detach(), Q.detach(), n, 0)
    g, = torch.autograd.grad(O.float().sum(), [xq])
    assert g.shape == xq.shape and torch.isfinite(g.float()).all() and float(g.float().abs().max()) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n,H,D,norm_from,weighted", [
    (1, 1, 8, 0, True),          # one row, one lane of the group at work
    (33, 5, 64, 10, True),       # one token beyond a CTA's 32, one head beyond a group of four
    (17, 4, 128, 0, True),       # one token beyond the 16 of a wide head
    (64, 12, 80, 64, True),      # nothing is normalised: the weight's gradient is zero
    (40, 3, 96, 0, False),       # rotation only
    (9473, 8, 64, 0, True),      # 594 tasks: two more than the CTAs, so two CTAs walk on
    (65, 2, 20, 5, True),        # a width without 16-byte accesses
])
def test_backward_kernel_matches_autograd_of_the_formulas(prep, n, H, D, norm_from, weighted, dtype):
    torch.manual_seed(n + D)
    x = torch.randn(n, H, D, device="cuda").to(dtype).requires_grad_(True)
    w = (1 + 0.1 * torch.randn(D, device="cuda")).to(dtype).requires_grad_(True) if weighted else None
    g = torch.randn(1, H, n, D, device="cuda").to(dtype)
    table = prep.rope_table(D, n + 3, device="cuda")
    wrt = [x, w] if weighted else [x]
    got = torch.autograd.grad(prep.qk_norm_rope(x, w, table, pos0=3, norm_from=norm_from), wrt, g)
    again = torch.autograd.grad(prep.qk_norm_rope(x, w, table, pos0=3, norm_from=norm_from), wrt, g, create_graph=True)
    x64 = x.detach().double().requires_grad_(True)
    w64 = w.detach().double().requires_grad_(True) if weighted else None
    # qk_norm_rope_torch works in fp32 inside: the formulas in fp64 instead
    y = x64
    if weighted:
        y = x64 * torch.rsqrt(x64.pow(2).mean(-1, keepdim=True) + 1e-6) * w64
        y = torch.where((torch.arange(n, device="cuda") < norm_from).view(n, 1, 1), x64, y)
    f = table[3:3 + n].double().unsqueeze(1)
    p = y.reshape(n, H, D // 2, 2)
    y = torch.stack([p[..., 0] * f[..., 0] - p[..., 1] * f[..., 1], p[..., 0] * f[..., 1] + p[..., 1] * f[..., 0]], -1)
    want = torch.autograd.grad(y.reshape(n, H, D).permute(1, 0, 2).unsqueeze(0), [x64, w64] if weighted else [x64], g.double())
    # results and the normalised factor are rounded to the type once each (unit roundoff u = 2^-9, 2^-12): 4 u of the
    # largest value; fp32 sums of up to n * H terms in a tree of 32-term chains: 1e-5
    tol = {torch.bfloat16: 2 ** -7, torch.float16: 2 ** -10, torch.float32: 1e-5}[dtype]
    for a, b, c in zip(got, again, want):
        assert a.dtype == dtype and a.shape == c.shape
        assert torch.equal(a, b.detach())
        assert float((a.double() - c).abs().max()) <= tol * float(c.abs().max()), (n, H, D)


@pytest.mark.gpu
def test_transforms_and_tracing_are_those_of_the_python_function(prep):
    """Forward mode and functorch transforms are refused by the call (a kernel called directly would drop
    the tangent); forward mode over its backward follows the formulas; torch.jit.trace records the call."""
    import torch.autograd.forward_ad as fwad
    torch.manual_seed(11)
    x, w = torch.randn(70, 3, 64, device="cuda"), 1 + 0.1 * torch.randn(64, device="cuda")
    table = prep.rope_table(64, 70, device="cuda")
    call = lambda a: prep.qk_norm_rope(a, w, table)
    for grad in (False, True):
        a = x.clone().requires_grad_(grad)
        with fwad.dual_level(), pytest.raises(RuntimeError):
            call(fwad.make_dual(a, torch.ones_like(a)))
    for transformed in (lambda: torch.func.jvp(call, (x,), (x,)), lambda: torch.func.vmap(call)(torch.stack([x, x]))):
        with pytest.raises(RuntimeError, match="functorch transforms"):
            transformed()
    u, du = torch.randn(1, 3, 70, 64, device="cuda"), torch.randn(1, 3, 70, 64, device="cuda")
    for keep in (False, True):
        a, b = (x.clone().requires_grad_(True) for _ in range(2))
        y = call(a)
        with fwad.dual_level():
            g, = torch.autograd.grad(y, [a], fwad.make_dual(u, du), create_graph=keep)
            got = fwad.unpack_dual(g).tangent
        want, = torch.autograd.grad(prep.qk_norm_rope_torch(b, w, table), [b], du)      # the backward is linear in g
        assert got is not None and torch.allclose(got, want, rtol=1e-4, atol=1e-5)
    for grad in (False, True):
        a = x.clone().requires_grad_(grad)
        traced = torch.jit.trace(call, (a,), check_trace=False)
        got, want = traced(a * 2), call(a * 2)
        assert torch.equal(got, want) and got.requires_grad == grad


@pytest.mark.gpu
def test_a_table_that_asks_for_gradients_is_accepted_and_gets_none(prep):
    table = prep.rope_table(64, 20, device="cuda").requires_grad_(True)
    y = prep.qk_norm_rope(torch.randn(20, 2, 64, device="cuda"), torch.ones(64, device="cuda"), table)
    y.sum().backward()
    assert y.requires_grad and table.grad is None


@pytest.mark.gpu
@pytest.mark.parametrize("n,H", [(70, 4), (64, 3), (70, 3)])      # tokens or heads that do not fill a CTA's tile
def test_backward_without_epsilon_is_finite(prep, n, H):
    torch.manual_seed(2)
    x = torch.randn(n, H, 64, device="cuda").requires_grad_(True)
    w = (1 + 0.1 * torch.randn(64, device="cuda")).requires_grad_(True)
    g, table = torch.randn(1, H, n, 64, device="cuda"), prep.rope_table(64, n, device="cuda")
    got = torch.autograd.grad(prep.qk_norm_rope(x, w, table, eps=0.0), [x, w], g)
    want = torch.autograd.grad(prep.qk_norm_rope_torch(x, w, table, eps=0.0), [x, w], g)
    for a, b in zip(got, want):      # fp32 on both sides
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-5 * float(b.abs().max()))
