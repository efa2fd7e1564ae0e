"""Decode path: split-K GEMM, paged attention, fused epilogues and the TP engine against dense f32 PyTorch evaluations."""
import math

import pytest
import torch

from ferrotorch_b200 import _lib, ops
from ferrotorch_b200.errors import FerrotorchError, IndexOutOfBounds, InvalidArgument
from ferrotorch_b200.models import LlamaConfig
from ferrotorch_b200.models.llama_infer import LlamaTPEngine, random_hf_weights, reference_last_logits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,splits", [(1280, 1024, 8), (520, 8192, 16), (256, 200, 3)])
def test_splitk_gemm_planes_sum_to_product(N, K, splits):
    torch.manual_seed(N + K)
    x = torch.zeros(16, K, device="cuda", dtype=torch.bfloat16)
    x[:5] = torch.randn(5, K, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, device="cuda").to(torch.bfloat16)
    planes = torch.full((splits, 16, N), float("nan"), device="cuda", dtype=torch.float32)
    _lib.call("ft_gemm_bf16_splitk", x, w, planes, 16, N, K, K, K, N, 0, 0, splits, _lib.S())
    ref = x.float() @ w.float().t()
    got = planes.sum(0)
    assert torch.isfinite(got).all()
    assert (got - ref).abs().max().item() <= 2e-3 * ref.abs().max().item() + 1e-3
    out = torch.empty(5, N, device="cuda", dtype=torch.bfloat16)
    _lib.call("ft_splitk_reduce", planes, splits, 5, N, N, 16 * N, None, out, N, 0, _lib.S())
    assert (out.float() - ref[:5]).abs().max().item() <= 2e-2 * ref.abs().max().item()


@pytest.mark.parametrize("Hq,Hkv,nsplit", [(8, 1, 4), (4, 2, 4), (2, 2, 4), (8, 1, 1), (8, 1, 13), (8, 1, 16), (8, 1, 37), (4, 2, 64)])
def test_paged_attention_decode(Hq, Hkv, nsplit):
    """Split counts on both sides of the combining pass's batch of sixteen, and more splits than a short sequence has pages (empty splits)."""
    torch.manual_seed(Hq * 10 + Hkv)
    B, D, max_blocks = 3, 128, 12
    lens = torch.tensor([1, 37, 160], device="cuda", dtype=torch.int32)
    nblk = B * max_blocks
    kc = torch.randn(nblk, 16, Hkv, D, device="cuda").to(torch.bfloat16)
    vc = torch.randn(nblk, 16, Hkv, D, device="cuda").to(torch.bfloat16)
    perm = torch.randperm(nblk, device="cuda").to(torch.int32).view(B, max_blocks).contiguous()     # scattered pages
    q = torch.randn(B, Hq, D, device="cuda").to(torch.bfloat16)
    out = torch.empty_like(q)
    ws = torch.zeros(B * Hkv * nsplit * (Hq // Hkv) * 132, device="cuda")
    ctr = torch.zeros(B * Hkv, device="cuda", dtype=torch.int32)
    for _ in range(2):      # second call checks that the counters reset themselves
        _lib.call("ft_paged_attn_decode", q, kc, vc, perm, max_blocks, lens, B, Hq, Hkv, D, 1.0 / math.sqrt(D), nsplit, ws, ctr, out, _lib.S())
    for b in range(B):
        n = int(lens[b])
        k = kc[perm[b].long()].reshape(-1, Hkv, D)[:n].float().repeat_interleave(Hq // Hkv, 1)
        v = vc[perm[b].long()].reshape(-1, Hkv, D)[:n].float().repeat_interleave(Hq // Hkv, 1)
        s = torch.einsum("hd,thd->ht", q[b].float(), k) / math.sqrt(D)
        ref = torch.einsum("ht,thd->hd", torch.softmax(s, -1), v)
        assert (out[b].float() - ref).abs().max().item() < 2e-2
    assert int(ctr.sum()) == 0


@pytest.mark.parametrize("use_graph", [False, True])
def test_tp_engine_single_gpu_matches_dense_reference(use_graph):
    cfg = LlamaConfig(vocab_size=1024, hidden_size=512, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=2, max_position_embeddings=256)
    W = random_hf_weights(cfg, "cuda", seed=1, std=0.05)
    eng = LlamaTPEngine(cfg, max_batch=4, max_seq=128, device="cuda", weights=W, use_graph=use_graph)
    torch.manual_seed(0)
    ids = torch.randint(0, cfg.vocab_size, (4, 40), device="cuda")
    seq = ids.clone()
    tok = eng.prefill(ids)
    ref = reference_last_logits(cfg, W, seq)
    assert (eng.logits - ref).abs().max().item() < 0.06 * ref.abs().max().item() + 0.02
    for _ in range(5):
        seq = torch.cat([seq, tok[:, None]], 1)
        tok = eng.decode_step().clone()
        ref = reference_last_logits(cfg, W, seq)
        assert (eng.logits - ref).abs().max().item() < 0.06 * ref.abs().max().item() + 0.02
    eng.check()


@pytest.mark.parametrize("layout", ["transposed", "columns", "offset", "shared", "padded", "short"])
@pytest.mark.parametrize("where", ["cuda", "cpu"])
def test_embedding_table_in_any_layout(layout, where):
    """The embedding table and the norm vectors as a program may hold them: prompt and decode steps read the rows of the table itself, in place or as a copy. Padded and short: more and
    fewer rows than the vocabulary (tokens of the rows that are there)."""
    cfg = LlamaConfig(vocab_size=512, hidden_size=256, intermediate_size=256, num_hidden_layers=1, num_attention_heads=2, num_key_value_heads=1, max_position_embeddings=64)
    W = {k: v.to(where, torch.bfloat16) for k, v in random_hf_weights(cfg, "cuda", seed=2, std=0.05).items()}
    e = W["model.embed_tokens.weight"]
    V, d = e.shape
    if layout == "transposed":
        odd = e.t().contiguous().t()
    elif layout == "columns":
        odd = torch.cat([torch.full_like(e, 9.0), e], 1)[:, d:]
    elif layout == "offset":
        odd = torch.cat([e.new_zeros(1), e.reshape(-1)])[1:].view(V, d)
    elif layout == "shared":
        odd = e = e[:1].expand(V, d)
    elif layout == "padded":
        odd = e = torch.cat([e, e.flip(0)[:8] * 2])
    else:
        odd = e = e[:40]
    plain, given = dict(W), dict(W)
    plain["model.embed_tokens.weight"], given["model.embed_tokens.weight"] = e.contiguous(), odd
    n = "model.layers.0.input_layernorm.weight"
    given[n] = torch.cat([W[n][:1], W[n]])[1:]                                    # a vector from an odd place
    engines = [LlamaTPEngine(cfg, max_batch=3, max_seq=64, device="cuda", weights=w, use_graph=False) for w in (plain, given)]
    ids = torch.randint(0, 40, (3, 20), device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    rows = engines[0].embed.shape[0]
    steps = torch.tensor([[0, 1, 39], [-1, -2, rows - 1], [-rows, 17, -3]], device="cuda")
    for eng in engines:
        eng.prefill(ids)
    assert torch.equal(engines[0].logits, engines[1].logits)
    full = plain["model.embed_tokens.weight"].cuda()
    for t in steps:
        for eng in engines:
            eng.tokens.copy_(t)
            eng.decode_step()
        assert torch.equal(engines[0].logits, engines[1].logits)
        seq = ids = torch.cat([ids, (t % rows)[:, None]], 1)
        ref = reference_last_logits(cfg, {**plain, "model.embed_tokens.weight": full}, seq)
        assert (engines[1].logits - ref).abs().max().item() < 0.06 * ref.abs().max().item() + 0.02
    engines[1].check()


@pytest.mark.parametrize("use_graph", [False, True])
def test_a_token_outside_the_table_stops_the_program(use_graph):
    cfg = LlamaConfig(vocab_size=512, hidden_size=256, intermediate_size=256, num_hidden_layers=1, num_attention_heads=2, num_key_value_heads=1, max_position_embeddings=64)
    W = random_hf_weights(cfg, "cuda", seed=2, std=0.05)
    ids = torch.randint(0, 40, (2, 20), device="cuda")
    eng, other = (LlamaTPEngine(cfg, max_batch=2, max_seq=64, device="cuda", weights=W, use_graph=use_graph) for _ in range(2))
    for resume in (eng.decode_step, lambda: eng.prefill(ids), eng.check):
        eng.prefill(ids)
        other.prefill(ids)
        eng.tokens.copy_(torch.tensor([3, 512]))
        eng.decode_step()
        torch.cuda.synchronize()
        other.decode_step()                                                       # another engine goes on
        with pytest.raises(IndexOutOfBounds, match="outside"):
            resume()
        assert resume == eng.check or _lib.read_status() >> 24 == 0x21
    want = other.generate(ids, 4)
    assert torch.equal(eng.generate(ids, 4), want)                                # and this one from its next prompt
    eng.check()
    few = LlamaTPEngine(cfg, max_batch=2, max_seq=64, device="cuda", weights={**W, "model.embed_tokens.weight": W["model.embed_tokens.weight"][:40]}, use_graph=use_graph)
    assert bool((want[:, :3] >= 40).any())
    with pytest.raises(IndexOutOfBounds):
        few.generate(ids, 4)
    with pytest.raises(IndexOutOfBounds):
        few.check()


def test_weights_that_do_not_fit_are_refused():
    cfg = LlamaConfig(vocab_size=512, hidden_size=256, intermediate_size=256, num_hidden_layers=1, num_attention_heads=2, num_key_value_heads=1, max_position_embeddings=64)
    W = random_hf_weights(cfg, "cuda", seed=2, std=0.05)
    for name, bad in (("model.embed_tokens.weight", torch.zeros(512, 264)), ("model.norm.weight", torch.ones(128))):
        with pytest.raises(InvalidArgument):
            LlamaTPEngine(cfg, max_batch=1, max_seq=64, device="cuda", weights={**W, name: bad})


def test_launchers_refuse_addresses_off_their_boundaries():
    t = torch.zeros(4096, device="cuda", dtype=torch.bfloat16)
    ids, planes = torch.zeros(1, device="cuda", dtype=torch.int64), torch.zeros(64, device="cuda")
    with pytest.raises(FerrotorchError):
        _lib.call("ft_decode_embed_norm", ids, t[1:], 4, t[1024:], t[2048:], t[3072:], 1, 64, 1e-5, _lib.S())
    with pytest.raises(FerrotorchError):
        _lib.call("ft_decode_residual_norm", planes[1:], 1, 4, 64, t, t[1024:], t[2048:], 1, 4, 1e-5, _lib.S())
    with pytest.raises(FerrotorchError):
        _lib.call("ft_decode_residual_norm", planes, 1, 4, 64, t[1:], t[1024:], t[2048:], 1, 4, 1e-5, _lib.S())
