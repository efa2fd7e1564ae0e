"""Gradient of the embedding table by id, in token order, and the scaling of prepared gradients: around the number of tokens that is looked through without sorting, ids that all
differ, repeat or lie outside the table."""
import pytest
import torch

from ferrotorch_b200 import _lib, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["random", "few", "one", "runs", "outside"])
@pytest.mark.parametrize("tokens,d", [(1, 8), (2, 4104), (131, 256), (-1, 1032), (0, 264), (1, 520), (5000, 8), (4500, 4104)])
def test_embedding_bwd_by_id(tokens, d, kind):
    tokens = _lib.kernels().ft_embedding_bwd_scan_max() + tokens if tokens <= 0 or (tokens, d) == (1, 520) else tokens
    torch.manual_seed(tokens + d)
    vocab = 997
    ids = torch.randint(0, {"random": vocab, "few": 3, "one": 1, "runs": vocab, "outside": vocab}[kind], (tokens,), device="cuda")
    if kind == "runs":                                      # every length up to 98 once, in any order of the tokens
        lengths = torch.arange(1, 100, device="cuda")
        ids = torch.repeat_interleave(torch.arange(99, device="cuda"), lengths)[torch.randperm(4950, device="cuda")].repeat(2)[:tokens]
    if kind == "outside":
        ids[::3] = vocab
        ids[1::5] = -1
    dout = torch.randn(tokens, d, device="cuda").bfloat16()
    for dtype in (torch.bfloat16, torch.float32):
        table = torch.randn(vocab, d, device="cuda").to(dtype)
        want = table.double()
        ok = (ids >= 0) & (ids < vocab)
        want.index_add_(0, ids[ok], dout[ok].double())
        got = ops.embedding_bwd(ids, dout, table.clone())
        # a row sums up to `tokens` terms in f32, each addition off by 2^-24 of a running sum of about sqrt(tokens); a bf16 table rounds the result once
        bound = tokens * tokens ** 0.5 * 2 ** -23 + (2 ** -8 * want.abs() if dtype == torch.bfloat16 else 0) + 1e-6
        assert ((got.double() - want).abs() <= bound).all()
        assert torch.equal(got, ops.embedding_bwd(ids, dout, table.clone()))


@pytest.mark.parametrize("tokens,d", [(1, 8), (131, 1032), (5000, 264)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_embedding_bwd_from_a_list_of_distinct_ids(tokens, d, dtype):
    """``ft_embedding_bwd_sorted`` of the C interface: the bits of the gradient by id."""
    torch.manual_seed(tokens + d)
    vocab = 97
    ids = torch.randint(-1, vocab + 1, (tokens,), device="cuda")
    dout, table = torch.randn(tokens, d, device="cuda").bfloat16(), torch.randn(vocab, d, device="cuda").to(dtype)
    sorted_ids, perm = torch.sort(ids, stable=True)
    uniq, counts = torch.unique_consecutive(sorted_ids, return_counts=True)
    got = table.clone()
    _lib.call("ft_embedding_bwd_sorted", uniq, torch.cumsum(counts, 0), perm, dout, got, uniq.numel(), d, vocab, int(dtype == torch.float32), _lib.S())
    assert torch.equal(got, ops.embedding_bwd(ids, dout, table.clone()))


@pytest.mark.parametrize("g", [1.0, 0.5, 1.0001, -3.0])
@pytest.mark.parametrize("n,m", [(8, 8), (8 * 1031, 64), (72, 8 * 70001), (12, 9)])
def test_scale_grads(n, m, g):
    torch.manual_seed(n)
    x, table, f = torch.randn(n, device="cuda").bfloat16(), torch.randn(m, device="cuda").bfloat16(), torch.tensor(g, device="cuda")
    want_x, want_t = x * f.bfloat16(), table * f.bfloat16()
    before = x.clone()
    out = ops.scale_grads(x, table, f)
    assert torch.equal(out, want_x) and torch.equal(table, want_t) and torch.equal(x, before)


@pytest.mark.parametrize("n", [0, 8, 8 * 1023, 8 * 1025, 8 * 70001, 12])
def test_zero(n):
    room = torch.full((n + 32,), 3.0, device="cuda").bfloat16()
    ops.zero_(room[16: 16 + n])
    assert (room[16: 16 + n] == 0).all() and (room[:16] == 3).all() and (room[16 + n:] == 3).all()
