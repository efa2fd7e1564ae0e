"""What the framework's speed is measured on: calls of its public entry points at the sizes that its configurations, benchmarks and tests use.

Kinds of cases:

* ``train``: a Llama decoder's forward pass, loss and backward pass (``LlamaForCausalLM(ids, labels=...)``, ``loss.backward()``), from the smoke test's sizes to
  two layers of the 8B configuration with its whole vocabulary;
* ``attention``: ``nn.functional.scaled_dot_product_attention`` as the encoders and any user's own module call it, forward alone or with its gradients;
* ``replay``: a prompt batch and the decoding of a given continuation on ``LlamaTPEngine`` (prompt pass, paged cache, captured decode step), logits of every step;
* ``serve``: requests of different lengths through ``ServingEngine.step`` for the Pufevik decoder: one ragged prompt batch, then single-token steps;
* ``conv``: one convolution layer of a ResNet trained under bf16 autocast, 32-bit weights, channels last, as ``bench_resnet.py`` trains fifty-three of them (alone: behind
  batch norms and rectifiers the rounding of 16-bit activations moves the gradients by more than any two kernels differ);
* ``update``: a step of ``AdamW`` or ``Sgd`` over the parameter tensors of a whole model.
"""
import math

import torch
import torch.nn.functional as F

from ferrotorch_b200 import nn, optim
from ferrotorch_b200.models import LlamaConfig, LlamaForCausalLM
from ferrotorch_b200.models.llama_infer import LlamaTPEngine
from ferrotorch_b200.models.pufevik import PufevikConfig, PufevikModel
from ferrotorch_b200.models.serving import ServingEngine, StepEntry
from ferrotorch_b200.vision.models import Conv1x1, Conv3x3

DEVICE = "cuda"
BF16 = torch.bfloat16

# Width, heads, key / value heads, feed-forward neurons, vocabulary: the smoke test's, the serving benchmark's three sizes (the largest with the 8B vocabulary).
LLAMA = {
    "smoke": (256, 2, 1, 512, 1024),
    "1k": (1024, 8, 2, 3072, 32768),
    "2k": (2048, 16, 4, 11264, 32768),
    "8b": (4096, 32, 8, 14336, 128256),
}
# Width, feed-forward neurons, heads, key / value heads, memory heads, memory key size, memory value size; window 1024, vocabulary 32768 (the serving benchmark's).
PUFEVIK = {
    "1k": (1024, 3072, 8, 2, 4, 128, 256),
    "2k": (2048, 11264, 16, 4, 4, 256, 512),
}
WINDOW, SERVE_VOCAB, GATE_CAP = 1024, 32768, 15.0
# Channels in and out, pixels per side, kernel, stride: layers of ResNet-50's four stages.
CONVS = {
    "stage1": (64, 64, 56, 3, 1), "stage1_expand": (64, 256, 56, 1, 1), "stage2_down": (128, 128, 56, 3, 2), "stage2": (128, 128, 28, 3, 1), "stage3": (256, 256, 14, 3, 1),
    "stage3_reduce": (1024, 256, 14, 1, 1), "stage4_shortcut": (1024, 2048, 14, 1, 2), "stage4": (512, 512, 7, 3, 1),
}


def listed():
    return [
        # the smallest training call: what a first run, a unit test or a search over hyperparameters does over and over; launches and host work count
        dict(name="train_smoke", kind="train", size="smoke", layers=2, batch=2, seq=64),
        # an ordinary fine-tuning batch with a length that divides nothing
        dict(name="train_1k_ragged", kind="train", size="1k", layers=2, batch=3, seq=777),
        # the pretraining step of the headline benchmark, two of its layers
        dict(name="train_8b", kind="train", size="8b", layers=2, batch=1, seq=4096),
        # self-attention of ViT-B/16 on a batch of 224 x 224 images (197 tokens), trained
        dict(name="attention_vit", kind="attention", batch=32, heads=12, kv_heads=12, seq=197, dim=64, causal=False, backward=True),
        # the encoder of Whisper on 30 seconds of audio (1500 frames), inference
        dict(name="attention_whisper", kind="attention", batch=4, heads=8, kv_heads=8, seq=1500, dim=64, causal=False, backward=False),
        # a long document through grouped-query attention, trained
        dict(name="attention_long", kind="attention", batch=1, heads=16, kv_heads=4, seq=6001, dim=128, causal=True, backward=True),
        # one user's short chat turn: latency of the prompt and of each token
        dict(name="replay_1k_short", kind="replay", size="1k", layers=2, batch=1, prompt=37, steps=24),
        # the decode benchmark's batch of eight prompts of 2048 tokens, four layers
        dict(name="replay_8b", kind="replay", size="8b", layers=4, batch=8, prompt=2048, steps=32),
        # three short requests of different lengths
        dict(name="serve_1k", kind="serve", size="1k", layers=2, sequences=3, longest=301, steps=16),
        # five longer requests, a few thousand tokens together
        dict(name="serve_2k", kind="serve", size="2k", layers=2, sequences=5, longest=1900, steps=16),
        # the 3 x 3 layer of the second stage on the training benchmark's batch
        dict(name="conv_28", kind="conv", layer="stage2", images=256),
        # the optimizer's step for a ResNet-50-like list: many small tensors, some large ones
        dict(name="update_many", kind="update", rule="adamw", dtype="f32", tensors=161, largest=2359296),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["train", "attention", "replay", "serve", "conv", "update"])
    if kind == "train":
        size = rng.choice(["smoke", "1k", "2k", "8b"])
        batch = rng.choice([1, 1, 2, 3])
        return dict(kind=kind, size=size, layers=rng.choice([1, 2]), batch=batch, seq=min(_log(rng, 17, 4096), 4096 // batch))
    if kind == "attention":
        kv = rng.choice([1, 2, 4, 8, 12])
        heads = kv * rng.choice([1, 1, 2, 4])
        seq = _log(rng, 33, 8192)
        batch = max(1, min(64, _log(rng, 1, 64), int(3.2e9 / (heads * seq * seq)), 400000 // (heads * seq)))
        return dict(kind=kind, batch=batch, heads=heads, kv_heads=kv, seq=seq, dim=rng.choice([32, 64, 64, 80, 96, 128, 128]), causal=rng.random() < 0.5,
                    backward=rng.random() < 0.6)
    if kind == "replay":
        return dict(kind=kind, size=rng.choice(["1k", "2k", "8b"]), layers=rng.choice([1, 2, 3, 4]), batch=rng.randint(1, 8), prompt=_log(rng, 17, 2048), steps=rng.randint(8, 32))
    if kind == "serve":
        return dict(kind=kind, size=rng.choice(["1k", "2k"]), layers=rng.choice([1, 2, 3, 4]), sequences=rng.randint(1, 6), longest=_log(rng, 20, 2000), steps=rng.randint(4, 16))
    if kind == "conv":
        return dict(kind=kind, layer=rng.choice(sorted(CONVS)), images=_log(rng, 4, 256))
    return dict(kind=kind, rule=rng.choice(["adamw", "sgd"]), dtype=rng.choice(["f32", "f32", "bf16"]), tensors=_log(rng, 8, 200), largest=_log(rng, 4096, 1 << 23))


# -- inputs -------------------------------------------------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _normal(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(shape, device=DEVICE, generator=g) * std).to(dtype)


def _tokens(g, vocab, *shape):
    return torch.randint(0, vocab, shape, device=DEVICE, generator=g)


def _llama_config(case):
    width, heads, kv, ff, vocab = LLAMA[case["size"]]
    return LlamaConfig(vocab_size=vocab, hidden_size=width, intermediate_size=ff, num_hidden_layers=case["layers"], num_attention_heads=heads, num_key_value_heads=kv)


def _llama_weights(case, g):
    """Random weights under the names of a checkpoint."""
    width, heads, kv, ff, vocab = LLAMA[case["size"]]
    D = width // heads
    mat = lambda o, i: _normal(g, o, i, std=0.02)                      # noqa: E731
    vec = lambda: (1 + 0.05 * torch.randn(width, device=DEVICE, generator=g)).to(BF16)  # noqa: E731
    w = {"model.embed_tokens.weight": mat(vocab, width), "lm_head.weight": mat(vocab, width), "model.norm.weight": vec()}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        w[p + "self_attn.q_proj.weight"] = mat(heads * D, width)
        w[p + "self_attn.k_proj.weight"] = mat(kv * D, width)
        w[p + "self_attn.v_proj.weight"] = mat(kv * D, width)
        w[p + "self_attn.o_proj.weight"] = mat(width, heads * D)
        w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"], w[p + "mlp.down_proj.weight"] = mat(ff, width), mat(ff, width), mat(width, ff)
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = vec(), vec()
    return w


def _llama_inputs(case, seed):
    g = _gen(seed)
    w, vocab = _llama_weights(case, g), LLAMA[case["size"]][4]
    if case["kind"] == "train":
        ids = _tokens(g, vocab, case["batch"], case["seq"] + 1)
        return w, ids[:, :-1].contiguous(), ids[:, 1:].contiguous()
    return w, _tokens(g, vocab, case["batch"], case["prompt"]), _tokens(g, vocab, case["steps"], case["batch"])


def _attention_inputs(case, seed):
    g, B, S, D = _gen(seed), case["batch"], case["seq"], case["dim"]
    return [_normal(g, B, S, n * D) for n in (case["heads"], case["kv_heads"], case["kv_heads"], case["heads"])]


def _pufevik_kinds(case):
    return ("pa" * case["layers"])[: case["layers"]]


def _pufevik_weights(case, g):
    width, ff, H, G, mh, md, mv = PUFEVIK[case["size"]]
    mat = lambda o, i: _normal(g, o, i, std=i ** -0.5)                 # noqa: E731
    vec = lambda n, mean=1.0, std=0.05: (mean + std * torch.randn(n, device=DEVICE, generator=g)).to(BF16)  # noqa: E731
    w = {"embed": mat(SERVE_VOCAB, width), "head": mat(SERVE_VOCAB, width), "final.norm": vec(width)}

    def attention(p, whole, gates):
        w.update({p + "q": mat(H * 128, width), p + "k": mat(G * 128, width), p + "v": mat(G * 128, width), p + "g": mat(gates, width), p + "o": mat(width, H * 128),
                  p + "q.norm": vec(H * 128 if whole else 128), p + "k.norm": vec(G * 128 if whole else 128)})
    for i, kind in enumerate(_pufevik_kinds(case)):
        p = f"l{i}."
        if kind == "a":
            attention(p + "mix.", False, H * 128)
            w[p + "mix.vmix"] = (0.5 + 0.1 * torch.randn((), device=DEVICE, generator=g)).to(BF16)
        else:
            attention(p + "mix.left.", True, H)
            q = p + "mix.right."
            w[p + "mix.left.sink"] = vec(H, 0.0, 1.0)
            w.update({q + "q": mat(mh * md, width), q + "k": mat(mh * md, width), q + "v": mat(mh * mv, width), q + "g": mat(mh * mv, width), q + "o": mat(width, mh * mv),
                      q + "norm": vec(mh * mv), q + "i": mat(mh, width), q + "f": mat(mh, width), q + "i.b": vec(mh, 0.0, 1.0), q + "f.b": vec(mh, 3.0, 1.0)})
        w.update({p + "norm1": vec(width), p + "norm2": vec(width), p + "mlp.gate": mat(ff, width), p + "mlp.up": mat(ff, width), p + "mlp.down": mat(width, ff)})
    return w


def _serve_lengths(case):
    """Prompt lengths: the longest one and shorter ones, none a multiple of another."""
    return [max(1, int(case["longest"] * (1.0, 0.31, 0.07, 0.77, 0.53, 0.19)[i])) for i in range(case["sequences"])]


def _serve_inputs(case, seed):
    g = _gen(seed)
    w = _pufevik_weights(case, g)
    return w, [_tokens(g, SERVE_VOCAB, n + case["steps"]).tolist() for n in _serve_lengths(case)]


def _conv_inputs(case, seed):
    cin, cout, side, k, stride = CONVS[case["layer"]]
    g, out = _gen(seed), (side + stride - 1) // stride
    w = _normal(g, cout, cin, k, k, std=math.sqrt(2.0 / (cout * k * k)), dtype=torch.float32)
    x = torch.relu(torch.randn(case["images"], cin, side, side, device=DEVICE, generator=g)).to(BF16)
    dy = _normal(g, case["images"], cout, out, out)
    return w, x.contiguous(memory_format=torch.channels_last), dy.contiguous(memory_format=torch.channels_last)


def _update_sizes(case):
    """Tensors of a network in its order: weights whose sizes go up and down between 64 and ``largest``, vectors in between."""
    top = math.log(case["largest"] / 64.0)
    return [64 * (i % 29 + 1) if i % 3 else int(64 * math.exp(top * (0.5 - 0.5 * math.cos(0.37 * i)))) // 8 * 8 + 8 * (i % 2) for i in range(case["tensors"])]


def _update_inputs(case, seed):
    g, dt = _gen(seed), torch.float32 if case["dtype"] == "f32" else BF16
    return [(_normal(g, n, std=0.02, dtype=dt), _normal(g, n, std=1e-3, dtype=dt)) for n in _update_sizes(case)]


# -- what a program has in hand before the call ---------------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "train":
        w, s["ids"], s["labels"] = _llama_inputs(case, seed)
        s["model"] = LlamaForCausalLM(_llama_config(case), device=DEVICE)
        s["model"].load_hf_state_dict(w)
    elif kind == "attention":
        s["q"], s["k"], s["v"], s["dout"] = _attention_inputs(case, seed)
        for t in (s["q"], s["k"], s["v"]):
            t.requires_grad_(case["backward"])
    elif kind == "replay":
        w, s["prompt"], s["tokens"] = _llama_inputs(case, seed)
        s["engine"] = LlamaTPEngine(_llama_config(case), max_batch=case["batch"], max_seq=case["prompt"] + case["steps"] + 1, device=DEVICE, weights=w)
    elif kind == "serve":
        w, s["tokens"] = _serve_inputs(case, seed)
        width, ff, H, G, mh, md, mv = PUFEVIK[case["size"]]
        cfg = PufevikConfig.pattern(_pufevik_kinds(case), SERVE_VOCAB, width, ff, H, G, 128, 128, WINDOW, mh, md, mv, gate_cap=GATE_CAP)
        room = sum(len(t) for t in s["tokens"]) + 16 * len(s["tokens"])
        s["engine"] = ServingEngine(PufevikModel(cfg, w, DEVICE), max_tokens=room, max_sequences=len(s["tokens"]))
    elif kind == "conv":
        cin, cout, _, k, stride = CONVS[case["layer"]]
        w, s["x"], s["dy"] = _conv_inputs(case, seed)
        s["conv"] = (Conv1x1 if k == 1 else Conv3x3)(cin, cout, stride).to(DEVICE)
        with torch.no_grad():
            s["conv"].weight.copy_(w)
        s["conv"] = s["conv"].to(memory_format=torch.channels_last)
        s["x"].requires_grad_(True)
    else:
        pairs = _update_inputs(case, seed)
        s["flat"] = torch.cat([p for p, _ in pairs])                   # the parameters lie one behind the other, as a flattened model's do
        s["params"] = [torch.nn.Parameter(p) for p in s["flat"].split([p.numel() for p, _ in pairs])]
        for p, (_, g) in zip(s["params"], pairs):
            p.grad = g
        s["opt"] = (optim.AdamW(s["params"], lr=3e-4, betas=(0.9, 0.95), weight_decay=0.1) if case["rule"] == "adamw"
                    else optim.Sgd(s["params"], lr=0.1, momentum=0.9, weight_decay=1e-4))
    return s


# -- one pass -------------------------------------------------------------------------------------------------------------------------------------------------------------
def run(s):
    return globals()["_run_" + s["case"]["kind"]](s["case"], s)


def _run_train(case, s):
    loss = s["model"](s["ids"], labels=s["labels"])
    loss.backward()
    return dict(loss=loss.detach(), grads=[u.views(u.grad) for u in s["model"].units()])


def _run_attention(case, s):
    B, S, D = case["batch"], case["seq"], case["dim"]
    q, k, v = (s[n].view(B, S, -1, D).transpose(1, 2) for n in "qkv")
    o = nn.functional.scaled_dot_product_attention(q, k, v, is_causal=case["causal"])
    o = o.transpose(1, 2).reshape(B, S, -1)
    if not case["backward"]:
        return dict(out=o)
    dq, dk, dv = torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["dout"])
    return dict(out=o.detach(), dq=dq, dk=dk, dv=dv)


def _run_replay(case, s):
    e = s["engine"]
    e.prefill(s["prompt"])
    logits = [e.logits.clone()]
    for t in s["tokens"]:
        e.tokens.copy_(t)
        e.decode_step()
        logits.append(e.logits.clone())
    return dict(logits=logits)


def _run_serve(case, s):
    e, lengths = s["engine"], _serve_lengths(case)
    ids = range(len(lengths))
    logits = [e.step([StepEntry(i, s["tokens"][i][: lengths[i]], [lengths[i] - 1]) for i in ids])]
    for k in range(case["steps"]):
        logits.append(e.step([StepEntry(i, [s["tokens"][i][lengths[i] + k]], [0]) for i in ids], ids if k + 1 == case["steps"] else ()))
    return dict(logits=logits)


def _run_conv(case, s):
    with torch.autocast("cuda", dtype=BF16):
        y = s["conv"](s["x"])
    dx, dw = torch.autograd.grad(y, (s["x"], s["conv"].weight), s["dy"])
    return dict(y=y.detach(), dx=dx, dw=dw)


def _run_update(case, s):
    s["opt"].step()
    return dict(params=s["flat"])


# -- what a pass cannot do without ----------------------------------------------------------------------------------------------------------------------------------------
def _llama_layer(case):
    """Weights of one layer and of the head, head size, heads, key / value heads, width, feed-forward neurons, vocabulary."""
    width, heads, kv, ff, vocab = LLAMA[case["size"]]
    D = width // heads
    return width * (heads + 2 * kv) * D + width * heads * D + 3 * width * ff, width * vocab, D, heads, kv, width, ff, vocab


def work(case):
    kind = case["kind"]
    if kind == "train":
        per, head, D, heads, kv, width, ff, vocab = _llama_layer(case)
        B, S, L = case["batch"], case["seq"], case["layers"]
        T = B * S
        pairs = B * heads * S * (S + 1) / 2
        # every product three times (output, input gradient, weight gradient); attention two products forward, five backward
        flops = 6 * T * (L * per + head) + L * pairs * D * 2 * 7
        # weights read, gradients written; the embedding's rows read once, its whole gradient written; the layers' inputs and outputs in both directions
        return dict(bytes=4 * (L * per + head) + 2 * vocab * width + 4 * T * width * (2 * L + 2), flops=flops)
    if kind == "attention":
        B, S, D, H, G = case["batch"], case["seq"], case["dim"], case["heads"], case["kv_heads"]
        pairs = B * H * (S * (S + 1) / 2 if case["causal"] else S * S)
        one = B * S * D * (2 * H + 2 * G) * 2                              # q, k, v in, output out
        return dict(bytes=one * (2.5 if case["backward"] else 1), flops=pairs * D * 2 * (7 if case["backward"] else 2))
    if kind == "replay":
        per, head, D, heads, kv, width, ff, vocab = _llama_layer(case)
        B, P, N, L = case["batch"], case["prompt"], case["steps"], case["layers"]
        cached = N * P + N * (N + 1) / 2                                   # rows of the cache that the steps of one sequence read
        flops = 2 * B * ((P + N) * L * per + (N + 1) * head) + 4 * B * L * heads * D * (P * (P + 1) / 2 + cached)
        return dict(bytes=(N + 1) * 2 * (L * per + head) + 4 * B * L * kv * D * (P + N + cached) + 4 * (N + 1) * B * vocab, flops=flops)
    if kind == "serve":
        width, ff, H, G, mh, md, mv = PUFEVIK[case["size"]]
        N, head = case["steps"], SERVE_VOCAB * width
        weights = flops = cache = 0
        for k in _pufevik_kinds(case):
            mix = width * 128 * (2 * H + 2 * G) + (width * H * 128 if k == "a" else width * (H + 2 * mh) + width * mh * (2 * md + 3 * mv))
            weights += mix + 3 * width * ff
            for n in _serve_lengths(case):
                seen = sum(min(t, WINDOW) if k == "p" else t for t in range(1, n + N + 1))
                flops += 2 * (n + N) * (mix + 3 * width * ff) + 4 * seen * H * 128 + (4 * (n + N) * mh * md * mv if k == "p" else 0)
                late = sum(min(t, WINDOW) if k == "p" else t for t in range(n + 1, n + N + 1))
                cache += 4 * G * 128 * (n + N + late) + (8 * N * mh * md * mv if k == "p" else 0)
        S = case["sequences"]
        return dict(bytes=(N + 1) * 2 * (weights + head) + cache + 4 * (N + 1) * S * SERVE_VOCAB, flops=flops + 2 * S * (N + 1) * head)
    if kind == "conv":
        cin, cout, side, k, stride = CONVS[case["layer"]]
        out = (side + stride - 1) // stride
        there, here = case["images"] * side * side * cin, case["images"] * out * out * cout
        # input, output gradient in; output, input gradient out; weight in, weight gradient out
        return dict(bytes=4 * (there + here) + 8 * cin * cout * k * k, flops=6 * here * cin * k * k)
    n = sum(_update_sizes(case))
    # 32-bit master and moments (momentum) in and out; the gradient in, 32 bits, or 16 and the 16-bit parameter out
    return dict(bytes=28 * n, flops=12 * n) if case["rule"] == "adamw" else dict(bytes=20 * n, flops=6 * n)


def tolerance(case):
    return {
        "train": dict(rel=0.03),
        "attention": dict(rel=0.01),
        "replay": dict(rel=0.03),
        "serve": dict(rel=0.03),
        "conv": dict(rel=0.01),
        "update": dict(rel=5e-7 if case.get("dtype") == "f32" else 2e-3),
    }[case["kind"]]


# -- the same in 64 bits --------------------------------------------------------------------------------------------------------------------------------------------------
def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)


def _rms(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _attend(q, k, v, causal, window=None, scale=None, sink=None):
    """``q`` ``[B, H, S, D]``, fewer heads in ``k`` and ``v``; one key / value head at a time."""
    S, R = q.shape[2], q.shape[1] // k.shape[1]
    hide = None
    if causal:
        back = torch.arange(S, device=q.device)[:, None] - torch.arange(S, device=q.device)
        hide = (back < 0) | (back >= (window or S))
    outs = []
    for g in range(k.shape[1]):
        s = q[:, g * R:(g + 1) * R] @ k[:, g:g + 1].transpose(-1, -2) * (scale or q.shape[-1] ** -0.5)
        if hide is not None:
            s = s.masked_fill(hide, -math.inf)
        if sink is not None:
            b = sink[g * R:(g + 1) * R].view(1, R, 1, 1).expand(s.shape[0], R, S, 1)
            p = torch.softmax(torch.cat([s, b], -1), -1)[..., :-1]
        else:
            p = torch.softmax(s, -1)
        outs.append(p @ v[:, g:g + 1])
    return torch.cat(outs, 1)


def _turn_halves(t, base):
    """``t`` ``[B, S, H, D]``: dimension i turns with i + D / 2."""
    S, D = t.shape[1], t.shape[3]
    a = torch.outer(torch.arange(S, device=t.device, dtype=torch.float64), base ** (-torch.arange(0, D, 2, device=t.device, dtype=torch.float64) / D))[None, :, None]
    u, v = t[..., : D // 2], t[..., D // 2:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def _llama_hidden(case, w, ids):
    width, heads, kv, ff, vocab = LLAMA[case["size"]]
    D, (B, S) = width // heads, ids.shape
    x = w["model.embed_tokens.weight"][ids]
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, w[p + "input_layernorm.weight"], 1e-5)
        q, k = (_turn_halves((h @ w[p + n + ".weight"].t()).view(B, S, -1, D), 500000.0).transpose(1, 2) for n in ("self_attn.q_proj", "self_attn.k_proj"))
        v = (h @ w[p + "self_attn.v_proj.weight"].t()).view(B, S, -1, D).transpose(1, 2)
        x = x + _attend(q, k, v, True).transpose(1, 2).reshape(B, S, heads * D) @ w[p + "self_attn.o_proj.weight"].t()
        h = _rms(x, w[p + "post_attention_layernorm.weight"], 1e-5)
        x = x + (F.silu(h @ w[p + "mlp.gate_proj.weight"].t()) * (h @ w[p + "mlp.up_proj.weight"].t())) @ w[p + "mlp.down_proj.weight"].t()
    return _rms(x, w["model.norm.weight"], 1e-5)


def _exact_train(case, seed):
    w, ids, labels = _llama_inputs(case, seed)
    w = {k: v.double().requires_grad_(True) for k, v in w.items()}
    h = _llama_hidden(case, w, ids)
    loss = F.cross_entropy(h.reshape(-1, h.shape[-1]) @ w["lm_head.weight"].t(), labels.reshape(-1))
    loss.backward()
    g = {k: v.grad for k, v in w.items()}
    units = [dict(weight=g["model.embed_tokens.weight"])]
    for i in range(case["layers"]):
        a, m, p = f"model.layers.{i}.self_attn.", f"model.layers.{i}.mlp.", f"model.layers.{i}."
        units.append(dict(norm1=g[p + "input_layernorm.weight"], norm2=g[p + "post_attention_layernorm.weight"],
                          wqkv=torch.cat([g[a + n + "_proj.weight"] for n in "qkv"]), wo=g[a + "o_proj.weight"],
                          wgu=torch.cat([g[m + "gate_proj.weight"], g[m + "up_proj.weight"]]), wd=g[m + "down_proj.weight"]))
    return dict(loss=loss.detach(), grads=units + [dict(weight=g["model.norm.weight"]), dict(weight=g["lm_head.weight"])])


def _exact_attention(case, seed):
    B, S, D = case["batch"], case["seq"], case["dim"]
    q, k, v, dout = (t.double() for t in _attention_inputs(case, seed))
    leaves = [t.requires_grad_(case["backward"]) for t in (q, k, v)]
    o = _attend(*(t.view(B, S, -1, D).transpose(1, 2) for t in leaves), case["causal"]).transpose(1, 2).reshape(B, S, -1)
    if not case["backward"]:
        return dict(out=o)
    dq, dk, dv = torch.autograd.grad(o, leaves, dout)
    return dict(out=o.detach(), dq=dq, dk=dk, dv=dv)


@torch.no_grad()
def _exact_replay(case, seed):
    w, prompt, tokens = _llama_inputs(case, seed)
    w = {k: v.double() for k, v in w.items()}
    h = torch.cat([_llama_hidden(case, w, row[None])[:, case["prompt"] - 1:] for row in torch.cat([prompt, tokens.t()], 1)])
    return dict(logits=[t.contiguous() for t in (h @ w["lm_head.weight"].t()).unbind(1)])


def _turn_pairs(t, dims, base):
    """``t`` ``[S, H, D]``: neighbouring dimensions below ``dims`` turn with one another."""
    a = torch.outer(torch.arange(t.shape[0], device=t.device, dtype=torch.float64), base ** (-torch.arange(0, dims, 2, device=t.device, dtype=torch.float64) / dims))[:, None]
    u, v = t[..., 0:dims:2], t[..., 1:dims:2]
    return torch.cat([torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2), t[..., dims:]], -1)


def _pufevik_memory(h, w, heads, dim, vdim, eps):
    """The gated recurrence token by token, all heads at once."""
    T = h.shape[0]
    cap = lambda z: GATE_CAP * torch.tanh(z / GATE_CAP)                # noqa: E731
    i, f = cap(h @ w["i"].t() + w["i.b"]), F.logsigmoid(cap(h @ w["f"].t() + w["f.b"]))
    q, k = (h @ w["q"].t()).view(T, heads, dim) * dim ** -0.5, (h @ w["k"].t()).view(T, heads, dim)
    v = (h @ w["v"].t()).view(T, heads, vdim)
    S, n, m = h.new_zeros(heads, dim, vdim), h.new_zeros(heads, dim), h.new_zeros(heads)
    out = torch.empty_like(v)
    for t in range(T):
        m2 = torch.maximum(f[t] + m, i[t])
        keep, add = torch.exp(f[t] + m - m2)[:, None], torch.exp(i[t] - m2)[:, None]
        S.mul_(keep[..., None]).add_((add * k[t])[..., None] * v[t][:, None])
        n, m = keep * n + add * k[t], m2
        out[t] = torch.einsum("hd,hdv->hv", q[t], S) / (torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
    o = out * torch.rsqrt(out.pow(2).mean(-1, keepdim=True) + eps)
    return (o.reshape(T, -1) * w["norm"] * torch.sigmoid(h @ w["g"].t())) @ w["o"].t()


@torch.no_grad()
def _exact_serve(case, seed):
    w, tokens = _serve_inputs(case, seed)
    w = {k: v.double() for k, v in w.items()}
    width, ff, H, G, mh, md, mv = PUFEVIK[case["size"]]
    eps, logits = 1e-6, []

    def attention(x, p, whole, window, sink):
        norm = lambda t, n: _rms(t, w[p + n], eps).view(x.shape[0], -1, 128) if whole else _rms(t.view(x.shape[0], -1, 128), w[p + n], eps)  # noqa: E731
        q, k = (_turn_pairs(norm(x @ w[p + n].t(), n + ".norm"), 64, 10000.0) for n in "qk")
        v = (x @ w[p + "v"].t()).view(-1, G, 128)
        return q, k, v
    for n, ids in zip(_serve_lengths(case), tokens):
        x, first = w["embed"][torch.tensor(ids, device=DEVICE)] * math.sqrt(width), None
        for i, kind in enumerate(_pufevik_kinds(case)):
            p = f"l{i}."
            a = p + ("mix." if kind == "a" else "mix.left.")
            q, k, v = attention(x, a, kind == "p", None, None)
            if kind == "a":
                if first is None:
                    first = v
                else:
                    v = (1 - w[a + "vmix"]) * v + w[a + "vmix"] * first
                o = _attend(q.transpose(0, 1)[None], k.transpose(0, 1)[None], v.transpose(0, 1)[None], True)[0].transpose(0, 1).reshape(x.shape[0], -1)
                y = (o * torch.sigmoid(x @ w[a + "g"].t())) @ w[a + "o"].t()
            else:
                o = _attend(q.transpose(0, 1)[None], k.transpose(0, 1)[None], v.transpose(0, 1)[None], True, WINDOW, None, w[a + "sink"])[0].transpose(0, 1)
                y = (o * torch.sigmoid(x @ w[a + "g"].t())[..., None]).reshape(x.shape[0], -1) @ w[a + "o"].t()
                r = p + "mix.right."
                y = y + _pufevik_memory(x, {n2[len(r):]: t for n2, t in w.items() if n2.startswith(r)}, mh, md, mv, eps)
            x = x + _rms(y, w[p + "norm1"], eps)
            y = (F.gelu(x @ w[p + "mlp.gate"].t(), approximate="tanh") * (x @ w[p + "mlp.up"].t())) @ w[p + "mlp.down"].t()
            x = x + _rms(y, w[p + "norm2"], eps)
        logits.append(_rms(x[n - 1:], w["final.norm"], eps) @ w["head"].t())
    return dict(logits=list(torch.stack(logits, 1)))


def _exact_conv(case, seed):
    w, x, dy = (t.double() for t in _conv_inputs(case, seed))
    k, stride = CONVS[case["layer"]][3:]
    x, w = x.requires_grad_(True), w.requires_grad_(True)
    y = F.conv2d(x, w, stride=stride, padding=k // 2)
    dx, dw = torch.autograd.grad(y, (x, w), dy)
    return dict(y=y.detach(), dx=dx, dw=dw)


@torch.no_grad()
def _exact_update(case, seed):
    values = []
    for p, g in _update_inputs(case, seed):
        p, g = p.double(), g.double()
        if case["rule"] == "adamw":
            p = p * (1 - 3e-4 * 0.1)
            m, v = 0.1 * g, 0.05 * g * g
            p = p - 3e-4 * (m / 0.1) / ((v / 0.05).sqrt() + 1e-8)
        else:
            p = p - 0.1 * (g + 1e-4 * p)
        values.append(p)
    return dict(params=torch.cat(values))
