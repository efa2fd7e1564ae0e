"""Backward RMSNorm around the widths where a row changes its number of threads and row counts around a CTA's rows; zero-padding of activations."""
import pytest
import torch

from ferrotorch_b200 import ops
from ferrotorch_b200.ops.conv import _padded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [8, 264, 1024, 1032, 2048, 2056, 4096, 4104])
@pytest.mark.parametrize("rows", [1, 3, 297, 1187])
@pytest.mark.parametrize("res", [False, True])
def test_rmsnorm_bwd(rows, d, res):
    torch.manual_seed(rows + d)
    x, dy, w = (torch.randn(*s, device="cuda").bfloat16() for s in ((rows, d), (rows, d), (d,)))
    dres = torch.randn(rows, d, device="cuda").bfloat16() if res else None
    _, rstd, _ = ops.rmsnorm_fwd(x, w, 1e-5)
    dx, dw = ops.rmsnorm_bwd(x, w, dy, rstd, dres=dres)
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    y = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    gx, gw = torch.autograd.grad(y, (xd, wd), dy.double())
    if res:
        gx = gx + dres.double()
    # one rounding to bf16, beside f32 arithmetic over `d` and `rows` terms
    assert ((dx.double() - gx).abs() <= 2 ** -8 * gx.abs() + 1e-4).all()
    assert ((dw.double() - gw).abs() <= 2 ** -8 * gw.abs() + 1e-5 * rows ** 0.5 + 1e-4).all()
    again, dw2 = ops.rmsnorm_bwd(x, w, dy, rstd, dres=dres)
    assert torch.equal(dx, again) and torch.equal(dw, dw2)


@pytest.mark.parametrize("d", [264, 1032, 4096, 4104])
@pytest.mark.parametrize("where", ["x", "dy", "dres"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_rmsnorm_bwd_row_that_is_not_finite(d, where, value):
    """One row with an element that is not finite: every other row keeps its bits, and so do the weight's gradients of columns where that row's product is unchanged (a gradient
    element that is not finite stays in its column)."""
    torch.manual_seed(d)
    rows, row, col = 37, 5, 9
    args = {n: torch.randn(rows, d, device="cuda").bfloat16() for n in ("x", "dy", "dres")}
    w = torch.randn(d, device="cuda").bfloat16()
    _, rstd, _ = ops.rmsnorm_fwd(args["x"], w, 1e-5)
    got = []
    for bad in (False, True):
        if bad:
            args[where][row, col] = value
        got.append(ops.rmsnorm_bwd(args["x"], w, args["dy"], rstd, dres=args["dres"]))
    (dx0, dw0), (dx1, dw1) = got
    others, columns = [r for r in range(rows) if r != row], [c for c in range(d) if c != col]
    assert torch.equal(dx0[others], dx1[others]) and not dx1[row, col].isfinite()
    assert torch.equal(dw0[columns], dw1[columns]) and dw1[col].isfinite() == (where == "dres")


@pytest.mark.parametrize("shape", [(1, 8, 1, 1), (2, 64, 7, 9), (3, 24, 28, 28)])
@pytest.mark.parametrize("pads", [(1, 1, 1, 1), (0, 0, 1, 1), (2, 0, 0, 3)])
def test_padded(shape, pads):
    t = torch.randn(shape, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    top, left, bottom, right = pads
    assert torch.equal(_padded(t, *pads), torch.nn.functional.pad(t.permute(0, 2, 3, 1), (0, 0, left, right, top, bottom)))
