"""What the performance of this package is measured on: the calls that a user's program makes, over
the range of sizes they are made with.

Three kinds of work, each through its public entry point:

* ``encode``: texts (token ids on the host) to embeddings (fp32 on the host) with
  ``eval.chunked_encoder.encode_chunked``, the call behind the MTEB wrapper, on a bf16 model built the
  way ``LSETMTEBModel.from_pretrained`` builds it (separate projections). Forward only.
* ``train``: one optimizer step from a collated, pinned host batch with
  ``TrainingEngine.train_step``: copy to the device, forward, loss, backward, clipping, AdamW.
  Returned are the loss and the updated fp32 weights.
* ``loss``: the contrastive loss of given embeddings with its gradients, on its own (InfoNCE with
  in-batch negatives, or a label matrix).

Model sizes are those of ``bench.py`` and the model configurations; the two wide ones are cut to a few
layers, so that several of them fit on a card. Weights are random, token ids are uniform, lengths are
uniform in a range: the work does not depend on their values.
"""
from __future__ import annotations

import math
import random

import torch

from lset_b200.eval.chunked_encoder import encode_chunked
from lset_b200.losses import fused_contrastive_loss, infonce_loss
from lset_b200.models import BertConfig, GemmaConfig, LlamaConfig, Qwen3Config, get_model_spec
from lset_b200.models.layers import init_normal_
from lset_b200.train.data.collator import LeftPadCollator, PackedCollator, RightPadCollator
from lset_b200.train.engine import TrainingEngine, pin

TEMPERATURE = 0.02
# Small enough for the loss of a second step on the same batch to be of the first one's size: at
# 2e-5 AdamW drives the loss of a batch of random texts to 1e-6 in one step, and nothing can be
# compared there. The work does not depend on it.
LR = 2e-6

# hidden, FFN, layers, query heads, KV heads, head dim, vocabulary
SIZES = {
    "qwen3-0.6b": ("qwen3", 1024, 3072, 28, 16, 8, 128, 151936),
    "qwen3-4b": ("qwen3", 2560, 9728, 36, 32, 8, 128, 151936),
    "qwen3-8b": ("qwen3", 4096, 12288, 36, 32, 8, 128, 151936),
    "llama-1b": ("llama", 2048, 8192, 16, 32, 8, 64, 128256),
    "embeddinggemma": ("embeddinggemma", 768, 1152, 24, 3, 1, 256, 262144),
    "bert-base": ("bert", 768, 3072, 12, 12, 12, 64, 30522),
}


def _encode(name, model, n, lo, hi, pooling="last_token"):
    return {"name": name, "kind": "encode", "model": model, "n": n, "lo": lo, "hi": hi,
            "pooling": pooling}


def _train(name, model, pairs, q, d, *, layers=0, negs=0, packed=True, lora=0, fp8=""):
    return {"name": name, "kind": "train", "model": model, "layers": layers or SIZES[model][3],
            "pairs": pairs, "q_lo": q[0], "q_hi": q[1], "d_lo": d[0], "d_hi": d[1], "negs": negs,
            "packed": packed, "lora": lora, "fp8": fp8}


def _loss(name, q, k, d, labels=False):
    return {"name": name, "kind": "loss", "q": q, "k": k, "d": d, "labels": labels}


def listed():
    return [
        # a search request: one query, where the latency of the call is what counts
        _encode("encode_one_query", "qwen3-0.6b", 1, 24, 40),
        # a request of several short texts to an encoder of the BERT kind
        _encode("encode_short_bert", "bert-base", 24, 8, 48, "mean"),
        # documents of an index, in token streams of the default budget
        _encode("encode_documents", "qwen3-0.6b", 128, 128, 512),
        # documents longer than a chunk: split, mean-pooled and merged
        _encode("encode_long_documents", "qwen3-0.6b", 10, 1500, 9000, "mean"),
        # the quick-start configuration: 8 pairs, padded batches, separate projections
        _train("train_quick", "qwen3-0.6b", 8, (8, 32), (32, 128), packed=False),
        # the headline of the benchmark: 64 pairs, packed, fused projections
        _train("train_packed", "qwen3-0.6b", 64, (16, 64), (128, 512)),
        # the bidirectional encoder of the comparison, mean pooling
        _train("train_bert", "bert-base", 8, (8, 32), (32, 128)),
        # adapters on a wide frozen model, hard negatives, recomputed activations
        _train("train_lora", "qwen3-8b", 16, (32, 32), (512, 512), layers=4, negs=3, lora=16),
        # 8-bit linear layers at the width where they pay
        _train("train_fp8", "qwen3-4b", 32, (16, 64), (256, 1024), layers=4, fp8="tensorwise"),
        # the loss at the smallest and at a large size of the loss benchmark
        _loss("loss_small", 1024, 1024, 768),
        _loss("loss_large", 8192, 8192, 1024),
        # a label matrix: one positive and three hard negatives per query, a ragged batch
        _loss("loss_labels", 1009, 4036, 1024, labels=True),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.499)))))))


def draw(rng: random.Random):
    kind = rng.choice(("encode", "encode", "train", "train", "loss"))
    if kind == "encode":
        model = rng.choice(("qwen3-0.6b", "qwen3-0.6b", "qwen3-0.6b", "bert-base", "bert-base",
                            "llama-1b", "embeddinggemma"))
        hi = _log(rng, 16, 512)
        n = _log(rng, 1, max(1, min(256, 40000 // hi)))
        case = _encode("", model, n, max(1, hi // rng.randint(1, 6)), hi,
                       rng.choice(("last_token", "mean", "mean")) if model != "bert-base" else "mean")
    elif kind == "train":
        model = rng.choice(("qwen3-0.6b", "qwen3-0.6b", "qwen3-0.6b", "bert-base", "qwen3-4b",
                            "qwen3-8b"))
        q_hi = _log(rng, 8, 64)
        d_hi = _log(rng, 32, 512)
        negs = rng.choice((0, 0, 1, 3)) if model != "bert-base" else 0
        pairs = _log(rng, 2, max(2, min(64, 20000 // ((1 + negs) * d_hi))))
        wide = model in ("qwen3-4b", "qwen3-8b")
        fp8 = "tensorwise" if model == "qwen3-4b" and rng.random() < 0.6 else ""
        case = _train("", model, pairs, (max(1, q_hi // 3), q_hi), (max(1, d_hi // 4), d_hi),
                      layers=rng.randint(1, 4) if wide else 0, negs=negs,
                      packed=model == "bert-base" or bool(fp8) or rng.random() < 0.7,
                      lora=rng.choice((8, 16)) if model == "qwen3-8b" else 0, fp8=fp8)
    else:
        labels = rng.random() < 0.4
        d = rng.choice((768, 1024, 1024, 2560, 4096))
        q = _log(rng, 16, 4096 if labels else 8192)
        k = q * rng.randint(1, 4)
        while q * k * d > 8192 * 8192 * 1024 or (labels and q * k > 2 ** 25):
            q = q * 2 // 3
            k = q * (k // q if k // q <= 4 else 4)
        case = _loss("", q, k, d, labels)
    del case["name"]
    return case


# --------------------------------------------------------------------------------------- models
def _config(case):
    family, h, ffn, layers, hq, hk, hd, vocab = SIZES[case["model"]]
    layers = case.get("layers") or layers
    if family == "bert":
        return family, BertConfig(vocab_size=vocab, hidden_size=h, intermediate_size=ffn,
                                  num_hidden_layers=layers, num_attention_heads=hq)
    cls = {"qwen3": Qwen3Config, "llama": LlamaConfig, "embeddinggemma": GemmaConfig}[family]
    kw = {}
    if family == "embeddinggemma":     # every sixth layer sees the whole sequence
        kw["layer_types"] = ["full_attention" if i % 6 == 5 else "sliding_attention"
                             for i in range(layers)]
    return family, cls(vocab_size=vocab, hidden_size=h, intermediate_size=ffn,
                       num_hidden_layers=layers, num_attention_heads=hq, num_key_value_heads=hk,
                       head_dim=hd, **kw)


def _texts(gen, n, lo, hi, vocab):
    lens = torch.randint(lo, hi + 1, (n,), generator=gen).tolist()
    flat = torch.randint(5, vocab, (sum(lens),), generator=gen).tolist()
    out, at = [], 0
    for m in lens:
        out.append(flat[at:at + m])
        at += m
    return out


def _as_ids(texts):
    return texts


def prepare(case, seed):
    gen = torch.Generator().manual_seed(seed)
    if case["kind"] == "loss":
        return _prepare_loss(case, seed)
    family, cfg = _config(case)
    spec = get_model_spec(family)
    if case["kind"] == "encode":
        torch.manual_seed(seed)
        with torch.device("cuda"):
            model = spec.model_cls(cfg)
        init_normal_(model, 0.02)
        model = model.to(torch.bfloat16).eval()
        return {"case": case, "model": model,
                "texts": _texts(gen, case["n"], case["lo"], case["hi"], cfg.vocab_size)}
    packed, bert = case["packed"], family == "bert"
    collator = PackedCollator() if packed else (RightPadCollator(0) if bert else LeftPadCollator(0))
    engine = TrainingEngine(
        family, None, dataset=None, collator=collator, batch_size=case["pairs"], lr=LR,
        max_steps=10 ** 9, grad_clip=1.0, temperature=0.05 if bert else TEMPERATURE, packed=packed,
        log_interval=0, scheduler_type="constant", model_config=cfg,
        fused_projections=packed and not case["lora"] and not bert,
        pooling="mean" if bert else "last_token", lora=case["lora"] > 0,
        lora_r=max(1, case["lora"]), lora_alpha=2.0 * case["lora"], fp8=bool(case["fp8"]),
        fp8_recipe=case["fp8"] or "tensorwise", activation_checkpoint=case["lora"] > 0,
        ac_mode="full", init_on_device=True, seed=seed)

    def sample(ids):
        return {"input_ids": ids, "attention_mask": [1] * len(ids)}

    P, vocab = case["pairs"], cfg.vocab_size
    q = _texts(gen, P, case["q_lo"], case["q_hi"], vocab)
    d = _texts(gen, P * (1 + case["negs"]), case["d_lo"], case["d_hi"], vocab)
    rows = []
    for i in range(P):
        row = {"query": sample(q[i]), "positive": sample(d[i])}
        if case["negs"]:
            lo = P + i * case["negs"]
            row["negatives"] = [sample(x) for x in d[lo:lo + case["negs"]]]
        rows.append(row)
    return {"case": case, "engine": engine, "batch": pin(collator(rows))}


def _prepare_loss(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def rows(n):
        x = torch.randn(n, case["d"], generator=gen, device="cuda")
        return torch.nn.functional.normalize(x, dim=1).to(torch.bfloat16).requires_grad_()

    state = {"case": case, "q": rows(case["q"]), "k": rows(case["k"])}
    if case["labels"]:
        Q, K = case["q"], case["k"]
        per = max(1, K // Q)
        qi = torch.arange(Q, device="cuda")
        labels = torch.zeros(Q, K, device="cuda")
        labels[qi, qi * per] = 1.0
        state.update(labels=labels, pos_qi=qi, pos_di=qi * per,
                     pos_counts=torch.ones(Q, dtype=torch.long, device="cuda"))
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "encode":
        return encode_chunked(state["model"], _as_ids, None, state["texts"], device="cuda",
                              pooling=case["pooling"])
    if case["kind"] == "train":
        engine = state["engine"]
        loss = engine.train_step(state["batch"])
        return [loss] + [g.master for g in engine.store.groups]
    q, k = state["q"], state["k"]
    if case["labels"]:
        loss = fused_contrastive_loss(q, k, state["labels"], TEMPERATURE, pos_qi=state["pos_qi"],
                                      pos_di=state["pos_di"], pos_counts=state["pos_counts"])
    else:
        loss = infonce_loss(q, k, TEMPERATURE)
    dq, dk = torch.autograd.grad(loss, (q, k))
    return [loss.detach(), dq, dk]


# ----------------------------------------------------------------------------------------- exact
def _rms64(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _attend64(q, k, v, scale, causal):
    """q [Hq, S, d], k and v [Hk, S, d] -> [S, Hq * d]; one KV head's group at a time."""
    groups, S = q.shape[0] // k.shape[0], q.shape[1]
    out = torch.empty_like(q)
    mask = torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1) if causal else None
    for h in range(k.shape[0]):
        rows = slice(h * groups, (h + 1) * groups)
        s = torch.matmul(q[rows], k[h].T) * scale
        if causal:
            s.masked_fill_(mask, -math.inf)
        out[rows] = torch.matmul(torch.softmax(s, -1), v[h])
    return out.transpose(0, 1).reshape(S, -1)


def _decoder64(w, cfg, causal, ids):
    S, d, half = ids.numel(), cfg.head_dim, cfg.head_dim // 2
    inv = cfg.rope_theta ** (-torch.arange(half, dtype=torch.float64, device="cuda") / half)
    angle = torch.outer(torch.arange(S, dtype=torch.float64, device="cuda"), inv)
    cos, sin = angle.cos(), angle.sin()

    def heads(x, n, norm):
        x = x.view(S, n, d)
        if norm is not None:
            x = _rms64(x, norm.double(), cfg.rms_norm_eps)
        return x.transpose(0, 1)

    def rotate(x):
        a, b = x[..., :half], x[..., half:]
        return torch.cat((a * cos - b * sin, b * cos + a * sin), -1)

    x = w["embed_tokens.weight"][ids].double()
    for i in range(cfg.num_hidden_layers):
        at = f"layers.{i}."

        def lin(y, name):
            return y @ w[at + name + ".weight"].double().T

        y = _rms64(x, w[at + "input_layernorm.weight"].double(), cfg.rms_norm_eps)
        q = heads(lin(y, "self_attn.q_proj"), cfg.num_attention_heads,
                  w.get(at + "self_attn.q_norm.weight"))
        k = heads(lin(y, "self_attn.k_proj"), cfg.num_key_value_heads,
                  w.get(at + "self_attn.k_norm.weight"))
        v = heads(lin(y, "self_attn.v_proj"), cfg.num_key_value_heads, None)
        o = _attend64(rotate(q), rotate(k), v, d ** -0.5, causal)
        x = x + lin(o, "self_attn.o_proj")
        y = _rms64(x, w[at + "post_attention_layernorm.weight"].double(), cfg.rms_norm_eps)
        y = torch.nn.functional.silu(lin(y, "mlp.gate_proj")) * lin(y, "mlp.up_proj")
        x = x + lin(y, "mlp.down_proj")
    return _rms64(x, w["norm.weight"].double(), cfg.rms_norm_eps)


def _bert64(w, cfg, ids):
    S, n, d = ids.numel(), cfg.num_attention_heads, cfg.hidden_size // cfg.num_attention_heads

    def lin(y, name):
        return y @ w[name + ".weight"].double().T + w[name + ".bias"].double()

    def norm(y, name):
        return torch.nn.functional.layer_norm(y, y.shape[-1:], w[name + ".weight"].double(),
                                              w[name + ".bias"].double(), cfg.layer_norm_eps)

    x = norm((w["embeddings.word_embeddings.weight"][ids].double()
              + w["embeddings.position_embeddings.weight"][:S].double()
              + w["embeddings.token_type_embeddings.weight"][0].double()), "embeddings.LayerNorm")
    for i in range(cfg.num_hidden_layers):
        at = f"layers.{i}."
        q, k, v = (lin(x, at + "attention." + p).view(S, n, d).transpose(0, 1)
                   for p in ("query", "key", "value"))
        o = _attend64(q, k, v, d ** -0.5, False)
        x = norm(x + lin(o, at + "attention.dense"), at + "attention.LayerNorm")
        y = torch.nn.functional.gelu(lin(x, at + "mlp.dense_in"))
        x = norm(x + lin(y, at + "mlp.dense_out"), at + "mlp.LayerNorm")
    return x


def _encode64(case, seed):
    if case["model"] == "embeddinggemma":   # four norms a block and two rotary bases: left out
        return None
    state = prepare(case, seed)
    family, cfg = _config(case)
    w = state["model"].state_dict()
    out = []
    for text in state["texts"]:
        total, acc = 0, 0.0
        for at in range(0, len(text), 4096 - 128):
            ids = torch.tensor(text[at:at + 4096], device="cuda")
            h = _bert64(w, cfg, ids) if family == "bert" else _decoder64(w, cfg, family == "qwen3",
                                                                         ids)
            emb = h[-1] if case["pooling"] == "last_token" else h.mean(0)
            acc, total = acc + emb * ids.numel(), total + ids.numel()
            if at + 4096 >= len(text):
                break
        out.append(torch.nn.functional.normalize(acc / total, dim=-1))
    return torch.stack(out).cpu().numpy()


@torch.no_grad()
def exact(case, seed):
    """The outputs of ``run`` in 64 bits. None for training steps: their loss is a single number and
    the updated weights are the old ones to six digits, so neither says how exact the step was."""
    if case["kind"] == "encode":
        return _encode64(case, seed)
    if case["kind"] == "train":
        return None
    state = _prepare_loss(case, seed)
    q, k = state["q"].double(), state["k"].double()
    rows = torch.arange(case["q"], device="cuda")
    target = state["pos_di"] if case["labels"] else rows
    p = (q @ k.T).div_(TEMPERATURE)      # one positive a row: cross entropy against its column
    lse = p.logsumexp(1)
    loss = (lse - p[rows, target]).mean()
    p.sub_(lse[:, None]).exp_()
    p[rows, target] -= 1.0
    p /= TEMPERATURE * case["q"]
    return [loss, p @ k, p.T @ q]


# ------------------------------------------------------------------------------------------ work
def _linear_params(case):
    family, h, ffn, layers, hq, hk, hd, _ = SIZES[case["model"]]
    layers = case.get("layers") or layers
    mlp = 2 * h * ffn if family == "bert" else 3 * h * ffn
    return layers, layers * (h * (hq + 2 * hk) * hd + hq * hd * h + mlp)


def _mean_square(lo, hi):
    n = hi - lo + 1
    return sum(x * x for x in range(lo, hi + 1)) / n


def work(case):
    if case["kind"] == "loss":
        q, k, d = case["q"], case["k"], case["d"]
        # scores once, and the two products with their gradient; embeddings in, gradients out
        return {"bytes": 4 * (q + k) * d + (4 * q * k if case["labels"] else 0),
                "flops": 6 * q * k * d}
    family, h, _, _, hq, _, hd, vocab = SIZES[case["model"]]
    layers, linear = _linear_params(case)
    causal = 0.5 if family in ("qwen3", "embeddinggemma") else 1.0
    if case["kind"] == "encode":
        n, lo, hi = case["n"], case["lo"], case["hi"]
        tokens = n * (lo + hi) / 2
        if hi <= 4096:
            squares = n * _mean_square(lo, hi)
        else:                           # chunks of 4096 tokens, 128 of them shared with the next
            squares = tokens * 3000
        attention = layers * 4 * causal * squares * hq * hd
        return {"bytes": 2 * linear + 2 * tokens * h + 4 * n * h,
                "flops": 2 * linear * tokens + attention}
    docs = case["pairs"] * (1 + case["negs"])
    tokens = (case["pairs"] * (case["q_lo"] + case["q_hi"]) + docs * (case["d_lo"] + case["d_hi"])) / 2
    squares = (case["pairs"] * _mean_square(case["q_lo"], case["q_hi"])
               + docs * _mean_square(case["d_lo"], case["d_hi"]))
    attention = layers * 4 * causal * squares * hq * hd * 3.5
    if case["lora"]:
        # frozen weights are read for forward and input gradients; their gradients are not formed
        return {"bytes": 2 * 2 * linear, "flops": 2 * 2 * linear * tokens + attention}
    # fp32 weights and two moments read and written, the bf16 copy of the weights written and read
    params = linear + vocab * h
    return {"bytes": 28 * params, "flops": 3 * 2 * linear * tokens + attention}


def tolerance(case):
    """Four times what was seen between this package's kernels and its eager attention, its eager
    norms and activations (losses: a computation in fp64), where 0.03 does not cap it. The
    gradients of a 28-layer bf16 model at temperature 0.02 differ by 2 % from one order of rounding
    to another (8-bit layers: 25 %) and most of it cancels in AdamW's quotient; what a step did to
    all of the weights shows in the loss of the step after it."""
    if case["kind"] == "encode":        # 28 layers, last token: 0.014 (largest value 0.08)
        return {"rel": 0.03, "max": 0.3}
    if case["kind"] == "loss":          # bf16 gradients of bf16 probabilities: 0.0018 (0.009)
        return {"rel": 0.008, "max": 0.04}
    if case["fp8"]:                     # the loss: 0.0077
        return {"rel": 0.03, "max": 0.06}
    return {"rel": 0.007, "max": 0.06}  # the loss: 0.0017; single weights: 0.0014
