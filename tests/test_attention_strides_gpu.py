"""Attention on operands read where they lie: head sizes around the kernels' 64 and 128 columns, lengths around their blocks, layouts that tile loads take and layouts that need a
copy, groups of query heads shared by a cluster; values and gradients against the f32 materialised form."""
import pytest
import torch

import ferrotorch_b200.nn as nn
from ferrotorch_b200.errors import InvalidArgument

pytestmark = pytest.mark.gpu

# bf16 operands and probabilities carry 2^-9 relative error each; sums over keys average it: 2 % of the norm bounds forward and backward
TOL = 2e-2


def _layout(kind, B, H, S, D):
    if kind == "heads":                                     # contiguous [B, H, S, D]
        return torch.randn(B, H, S, D, device="cuda").bfloat16()
    if kind == "rows":                                      # a projection's [B, S, H * D]
        return torch.randn(B, S, H * D, device="cuda").bfloat16().view(B, S, H, D).transpose(1, 2)
    if kind == "slice":                                     # columns of a wider row
        return torch.randn(B, S, H, D + 8, device="cuda").bfloat16()[..., 8:].transpose(1, 2)
    if kind == "odd":                                       # rows off the 16-byte boundaries
        return torch.randn(B, H, S, D + 1, device="cuda").bfloat16()[..., 1:]
    if kind == "shared":                                    # one head seen as all of them
        return torch.randn(B, 1, S, D, device="cuda").bfloat16().expand(B, H, S, D)
    return torch.randn(B, H, D, S, device="cuda").bfloat16().transpose(2, 3)


@pytest.mark.parametrize("kinds", [("heads", "rows", "slice"), ("rows", "odd", "columns"), ("slice", "shared", "heads")])
@pytest.mark.parametrize("B,Hq,Hkv,S,D,causal", [(1, 1, 1, 1, 8, True), (2, 3, 1, 63, 64, True), (1, 4, 2, 64, 72, False), (2, 2, 2, 65, 56, False), (1, 4, 1, 127, 128, True),
                                                 (3, 4, 4, 129, 64, True), (1, 8, 2, 193, 80, True), (1, 8, 1, 640, 128, True), (1, 6, 3, 257, 32, False)])
def test_strided_attention(B, Hq, Hkv, S, D, causal, kinds):
    if ops_backend() != "tcgen05":
        pytest.skip("native attention kernels not built")
    torch.manual_seed(S + D)
    q, k, v = (_layout(kind, B, h, S, D).requires_grad_() for kind, h in zip(kinds, (Hq, Hkv, Hkv)))
    qf, kf, vf = (t.detach().double().requires_grad_() for t in (q, k, v))
    o = nn.functional.scaled_dot_product_attention(q, k, v, is_causal=causal)
    ref = nn.standard_attention(qf, nn.repeat_kv(kf, Hq // Hkv), nn.repeat_kv(vf, Hq // Hkv), causal)
    g = torch.randn(B, S, Hq, D, device="cuda").bfloat16().transpose(1, 2)
    got, want = torch.autograd.grad(o, (q, k, v), g), torch.autograd.grad(ref, (qf, kf, vf), g.double())
    assert o.shape == (B, Hq, S, D)
    assert (o.double() - ref).norm() <= TOL * ref.norm()
    # single keys: the gradients of q and k are sums of differences that cancel, so their error is measured against the gradient's scale without cancellation
    floor = 1e-2 * g.double().norm() if S > 1 else 0.1 * g.double().norm()
    for a, b in zip(got, want):
        assert a.shape == b.shape and (a.double() - b).norm() <= TOL * b.norm() + 2e-2 * floor


@pytest.mark.parametrize("S", [65, 128, 129, 192, 500, 1000])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_scores_whose_maximum_stays(S, D, causal):
    """Equal scores: the accumulator is never rescaled behind the first block, and the output is the mean of the values in sight. Enough heads for several waves of CTAs."""
    if ops_backend() != "tcgen05":
        pytest.skip("native attention kernels not built")
    torch.manual_seed(S + D)
    q, k = torch.zeros(4, 64, S, D, device="cuda", dtype=torch.bfloat16), torch.randn(4, 64, S, D, device="cuda").bfloat16()
    v = torch.randn(4, 64, S, D, device="cuda").bfloat16()
    o = nn.functional.scaled_dot_product_attention(q, k, v, is_causal=causal)
    n = torch.arange(1, S + 1, device="cuda", dtype=torch.float64)[:, None]
    want = v.double().cumsum(2) / n if causal else v.double().mean(2, keepdim=True).expand(4, 64, S, D)
    # probabilities of one: the products are exact, their f32 sums are off by far less than the output's rounding of 2^-9
    assert ((o.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5).all()


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("B,Hq,Hkv,S,D,row", [(2, 2, 2, 197, 64, 70), (1, 4, 1, 300, 128, 0), (1, 2, 1, 640, 80, 129), (1, 2, 2, 100, 40, 63)])
def test_a_query_that_is_not_finite_stays_out_of_keys_it_does_not_see(B, Hq, Hkv, S, D, row, value):
    """Causal: the gradients of values behind query ``row``, and those of every other query, do not depend on it, so they keep their bits. (The gradients of keys are products with the
    query itself.)"""
    if ops_backend() != "tcgen05":
        pytest.skip("native attention kernels not built")
    torch.manual_seed(S + D)
    q, k, v = (torch.randn(B, h, S, D, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv))
    g = torch.randn(B, Hq, S, D, device="cuda").bfloat16()
    bad = q.clone()
    bad[:, :, row] = value
    got = []
    for x in (q, bad):
        leaves = [t.clone().requires_grad_() for t in (x, k, v)]
        o = nn.functional.scaled_dot_product_attention(*leaves, is_causal=True)
        got.append((o.detach(), *torch.autograd.grad(o, leaves, g)))
    (o0, dq0, _, dv0), (o1, dq1, _, dv1) = got
    others = [r for r in range(S) if r != row]
    assert torch.equal(o0[:, :, others], o1[:, :, others]) and torch.equal(dq0[:, :, others], dq1[:, :, others])
    assert torch.equal(dv0[:, :, row + 1:], dv1[:, :, row + 1:])


def ops_backend():
    from ferrotorch_b200 import ops
    return ops.attention.backend()


@pytest.mark.parametrize("refused", ["batch", "heads", "device"])
def test_operands_that_do_not_fit_are_refused(refused):
    q = torch.zeros(2, 4, 16, 64, device="cuda", dtype=torch.bfloat16)
    k = v = torch.zeros(1 if refused == "batch" else 2, 2, 16, 64, device="cpu" if refused == "device" else "cuda", dtype=torch.bfloat16)
    if refused == "heads":
        v = torch.zeros(2, 4, 16, 64, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(InvalidArgument):
        nn.functional.scaled_dot_product_attention(q, k, v)
