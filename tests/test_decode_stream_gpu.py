"""Kernels of a decode step on one GPU: the weight stream, the embedding with its norm, the residual update and the choice of the next token."""
import pytest
import torch

from ferrotorch_b200 import _lib
from ferrotorch_b200.models.llama_infer import LogitsPick, _SplitKGemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 7, 16])
@pytest.mark.parametrize("N,K", [(1, 8), (127, 64), (129, 72), (1536, 1024), (4, 20000), (640, 4104), (38000, 256)])
def test_weight_stream(N, K, rows):
    torch.manual_seed(N + K)
    x, w = torch.randn(16, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    g = _SplitKGemm(w, "cuda")
    g.planes.fill_(float("nan"))
    g(x, rows)
    got, want = g.planes[:, :rows, :N].sum(0).double(), x[:rows].double() @ w.double().t()
    # f32 sums of K products of unit normals: each addition rounds a running sum of about sqrt(K)
    assert (got - want).abs().max() <= 2 ** -23 * K * K ** 0.5 + 1e-6
    assert torch.isnan(g.planes[:, rows:]).all() and torch.isnan(g.planes[:, :, N:]).all()


@pytest.mark.parametrize("splits,rows,d", [(1, 1, 4), (3, 2, 100), (9, 16, 1024), (17, 5, 8200)])
def test_residual_norm(splits, rows, d):
    torch.manual_seed(d)
    ldp = (d + 3) // 4 * 4
    planes, x, w = torch.randn(splits, 16, ldp, device="cuda"), torch.randn(rows, d, device="cuda").bfloat16(), torch.randn(d, device="cuda").bfloat16()
    want_x = planes[:, :rows, :d].double().sum(0) + x.double()
    h = torch.empty_like(x)
    _lib.call("ft_decode_residual_norm", planes, splits, ldp, 16 * ldp, x, w, h, rows, d, 1e-5, _lib.S())
    assert (x.double() - want_x).abs().max() <= 2 ** -8 * want_x.abs().max()
    want_h = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    assert (h.double() - want_h).abs().max() <= 2 ** -8 * want_h.abs().max()


@pytest.mark.parametrize("splits,rows,N", [(1, 1, 1), (2, 3, 1027), (9, 16, 32768), (2, 8, 128256)])
def test_logits_pick(splits, rows, N):
    torch.manual_seed(N)
    ldp = (N + 3) // 4 * 4
    g = _SplitKGemm(torch.zeros(N, 8, device="cuda", dtype=torch.bfloat16), "cuda")
    g.planes, g.splits, g.plane_stride = torch.randn(splits, 16, ldp, device="cuda").round(decimals=1), splits, 16 * ldp
    if N > 2000:
        g.planes[:, 0, 1999] = g.planes[:, 0, 77] = 50.0                            # equal ones: the first
        g.planes[0, 1, 1234] = g.planes[0, 1, 9] = float("nan")
        g.planes[:, 2] = -0.0
        g.planes[:, 2, 5] = 0.0
    logits = torch.empty(rows, ldp, device="cuda")
    pick = LogitsPick(16, "cuda")
    tokens, picked = torch.full((rows,), -5, device="cuda"), torch.full((rows,), -5, device="cuda")
    pos = torch.arange(rows, device="cuda", dtype=torch.int32)
    lens = pos + 1
    for step in range(2):
        pick(g, logits, rows, N, tokens, picked, pos, lens)
        want = logits[:, :N].cpu().max(-1)
        assert torch.equal(tokens.cpu(), want.indices) and torch.equal(tokens, picked)
        assert pos.tolist() == [r + step + 1 for r in range(rows)] and lens.tolist() == [r + step + 2 for r in range(rows)]
        assert (pick.ws == 0).all()
    ref = g.planes[:, :rows, :N].double().sum(0)
    assert torch.allclose(logits[:, :N].double(), ref, rtol=1e-5, atol=1e-5, equal_nan=True)


def test_embed_norm():
    torch.manual_seed(0)
    table, w = torch.randn(50, 264, device="cuda").bfloat16(), torch.randn(264, device="cuda").bfloat16()
    tokens = torch.tensor([3, 49, -1, 0], device="cuda")
    x, h = torch.empty(4, 264, device="cuda", dtype=torch.bfloat16), torch.empty(4, 264, device="cuda", dtype=torch.bfloat16)
    _lib.call("ft_decode_embed_norm", tokens, table, 50, w, x, h, 4, 264, 1e-5, _lib.S())
    assert torch.equal(x, table[tokens])
    want = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    assert (h.double() - want).abs().max() <= 2 ** -8 * want.abs().max()
    outside = torch.tensor([50], device="cuda")
    _lib.call("ft_decode_embed_norm", outside, table, 50, w, x, h, 1, 264, 1e-5, _lib.S())
    assert (x[0] == 0).all() and (h[0] == 0).all() and _lib.read_status() >> 24 == 0x21
