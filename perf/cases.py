"""What a user of this package has it do, as cases that can be timed: the three
encoder stacks through the calls an embedding service makes (bucketed plans over
token lists, one captured plan over pinned host buffers, the native runner, packed
rows), the cached attention of a decoding step, the f32 attention with its
log-sum-exp and a single projection.

`listed()` are the fixed cases, `draw` makes more of the same ranges. A case is a
dict of plain values; `prepare` makes what a program holds before the call (model,
plans, host or device inputs), `run` is one call. Models are random-init, ids
uniform over the vocabulary, row lengths spread evenly from `shortest` to `longest`
and dealt in an order the seed gives, so a case is the same amount of work for
every seed.
"""
import math

import numpy as np
import torch

from svod_b200 import encoders as E
from svod_b200 import ops
from svod_b200.encoder_head import HeadPlans, Qwen3PackedEmbedder, plan_shape
from svod_b200.native import NativeModernBert, NativeQwen3, NativeXlmRoberta

XLMR, QWEN3, MODERNBERT = E.XlmRobertaConfig, E.Qwen3Config, E.ModernBertConfig
STACKS = {
    "xlmr": (XLMR, E.XlmRobertaEncoder, NativeXlmRoberta),
    "qwen3": (QWEN3, E.Qwen3Embedder, NativeQwen3),
    "modernbert": (MODERNBERT, E.ModernBertEncoder, NativeModernBert),
}
DTYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}


def listed():
    return [
        # One search query embedded while somebody waits: the smallest call a service makes.
        dict(name="xlmr_query", path="heads", model="xlmr", rows=1, shortest=21, longest=21),
        # The same for the decoder-style embedder, from compiled code, at the caller's own odd length.
        dict(name="qwen3_query", path="native", model="qwen3", rows=1, shortest=43, longest=43),
        # A handful of paragraphs of unequal length, mean-pooled: an interactive batch.
        dict(name="modernbert_paragraphs", path="heads", model="modernbert", rows=7, shortest=35, longest=301),
        # Indexing passages: a full batch with the usual mix of lengths and padding.
        dict(name="xlmr_passages", path="heads", model="xlmr", rows=64, shortest=64, longest=512),
        # Many short and medium texts packed end to end into shared rows.
        dict(name="qwen3_packed", path="packed", model="qwen3", texts=120, shortest=12, longest=1000, max_batch=8),
        # Long documents, windowed and global layers, padded to the longest.
        dict(name="modernbert_documents", path="plan", model="modernbert", rows=16, shortest=2048, longest=8192),
        # The throughput job of the embedder: full-length rows, the largest case.
        dict(name="qwen3_documents", path="plan", model="qwen3", rows=32, shortest=4096, longest=4096),
        # One decoding step of a few long conversations: a cache read once per step.
        dict(name="decode_long_cache", path="decode", dtype="bfloat16", batch=8, queries=1, cache=32768, shortest=30000,
             heads=16, kv_heads=8, head_dim=128, appended=0),
        # A decoding step of a wide batch in a shared cache (row map), the newest tokens not in it yet.
        dict(name="decode_appended", path="decode", dtype="float16", batch=24, queries=1, cache=2048, shortest=150,
             heads=16, kv_heads=8, head_dim=64, appended=5),
        # f32 attention with key lengths and log-sum-exp: the checking configuration.
        dict(name="attention_f32", path="attention", dtype="float32", batch=2, queries=512, cache=512, shortest=256,
             heads=8, kv_heads=8, head_dim=64),
        # One projection of a short batch: ragged rows, bias and activation in the store.
        dict(name="linear_short", path="linear", dtype="bfloat16", m=509, n=1024, k=1024, act="gelu", gated=False,
             bias=True, residual=False),
        # A gated projection of a medium batch.
        dict(name="linear_gated", path="linear", dtype="bfloat16", m=4000, n=3072, k=1024, act="silu", gated=True,
             bias=False, residual=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["model", "model", "model", "packed", "decode", "decode", "attention", "linear", "linear"])
    if path == "model":
        model = rng.choice(["xlmr", "qwen3", "modernbert"])
        most_rows, most_len = {"xlmr": (64, 512), "qwen3": (32, 4096), "modernbert": (16, 8192)}[model]
        longest = _log(rng, 16, most_len)
        how = {"xlmr": ["heads", "heads", "native"], "modernbert": ["heads", "plan", "native"], "qwen3": ["plan", "native"]}
        return dict(path=rng.choice(how[model]), model=model, rows=_log(rng, 1, most_rows),
                    shortest=max(1, int(longest * rng.uniform(0.1, 1.0))), longest=longest)
    if path == "packed":
        longest = _log(rng, 60, 2000)
        return dict(path="packed", model="qwen3", texts=_log(rng, 4, 150), shortest=rng.randint(3, longest // 2),
                    longest=longest, max_batch=rng.choice([4, 8, 16]))
    if path == "decode":
        batch = _log(rng, 1, 64)
        cache = _log(rng, 200, min(32768, 262144 // batch))
        head_dim, kv_heads, group = rng.choice([64, 128]), rng.choice([4, 8, 16]), rng.choice([1, 2, 4])
        return dict(path="decode", dtype=rng.choice(["bfloat16", "float16"]), batch=batch, queries=rng.choice([1, 1, 1, 4, 16]),
                    cache=cache, shortest=max(1, int(cache * rng.uniform(0.1, 1.0))), heads=kv_heads * group,
                    kv_heads=kv_heads, head_dim=head_dim, appended=rng.choice([0, 0, 1, 5, 16]))
    if path == "attention":
        tokens = _log(rng, 50, 1024)
        return dict(path="attention", dtype="float32", batch=rng.randint(1, 4), queries=tokens, cache=tokens,
                    shortest=max(1, tokens // 2), heads=8, kv_heads=rng.choice([4, 8]), head_dim=rng.choice([64, 128]))
    gated = rng.random() < 0.4
    act = "silu" if gated else rng.choice(["none", "gelu", "gelu_tanh"])
    return dict(path="linear", dtype=rng.choice(["bfloat16", "float16"]), m=_log(rng, 20, 32768),
                n=rng.choice([768, 1024, 3072, 4096]), k=rng.choice([768, 1024, 3072, 4096]), act=act, gated=gated,
                bias=rng.random() < 0.5, residual=act == "none" and rng.random() < 0.5)


# ------------------------------------------------------------------------------------ inputs
def _lengths(n, shortest, longest):
    return [int(round(shortest + (longest - shortest) * (i + 1) / n)) if n > 1 else longest for i in range(n)]


def _texts(case, n, vocab, seed):
    """`n` token lists, ids uniform over the vocabulary past the special ones."""
    r = np.random.RandomState(seed % (1 << 32))
    lens = _lengths(n, case["shortest"], case["longest"])
    r.shuffle(lens)
    return [r.randint(5, vocab, k).tolist() for k in lens]


def _pinned(case, texts, rows, length, mask):
    """Host buffers of a plan: padded ids, the padding mask or the lengths."""
    ids = torch.full((rows, length), 1, dtype=torch.int32).pin_memory()
    aux = torch.zeros(rows, length, dtype=torch.bool) if mask else torch.zeros(rows, dtype=torch.int32)
    for i, t in enumerate(texts):
        ids[i, :len(t)] = torch.tensor(t, dtype=torch.int32)
        if mask:
            aux[i, :len(t)] = True
        else:
            aux[i] = len(t)
    return ids, aux.pin_memory()


def _prepare_model(case, seed):
    config, stack, native = STACKS[case["model"]]
    cfg = config()
    model = stack.random_init(cfg, seed=seed)
    path = case["path"]
    if path == "packed":
        texts = _texts(case, case["texts"], cfg.vocab_size, seed)
        return dict(texts=texts, embedder=Qwen3PackedEmbedder(model, case["max_batch"], case["longest"]))
    texts = _texts(case, case["rows"], cfg.vocab_size, seed)
    if path == "heads":
        plans = HeadPlans(model, max_batch=64)
        # the service has warmed its plans up with a batch of this shape
        plans.run([[7] * case["longest"]] * case["rows"])
        return dict(plans=plans, texts=texts)
    mask = case["model"] != "qwen3"
    if path == "native":
        ids, aux = _pinned(case, texts, case["rows"], case["longest"], mask)
        runner = native(model)
        runner.plan(case["rows"], case["longest"])
        out = torch.empty(case["rows"], cfg.hidden_size).pin_memory()
        return dict(runner=runner, keep=(ids, aux, out), ids=ids.numpy(), out=out.numpy(),
                    aux=(aux.view(torch.uint8) if mask else aux).numpy())
    rows, length = plan_shape(case["rows"], case["longest"], case["rows"])
    ids, aux = _pinned(case, texts, rows, length, mask)
    plan = E.Plan(model, rows, length, "mask" if mask else "lengths").capture()
    return dict(plan=plan, ids=ids, aux=aux, out=torch.empty(rows, cfg.hidden_size).pin_memory())


def _prepare_attention(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    B, T, Tk, H, Hk, D = (case[k] for k in ("batch", "queries", "cache", "heads", "kv_heads", "head_dim"))
    n = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=dt)
    lens = _lengths(B, case["shortest"], Tk)
    np.random.RandomState(seed % (1 << 32)).shuffle(lens)
    keys = ops.KeyMask.Lens(torch.tensor(lens, dtype=torch.int32, device="cuda"))
    q, k, v = n(B, T, H, D), n(B, Tk, Hk, D), n(B, Tk, Hk, D)
    if case["path"] == "attention":
        return dict(q=q, k=k, v=v, opts=ops.Attn(keys=keys, want_lse=True))
    cache = None
    if case["appended"]:
        rows = torch.randperm(B, generator=g, device="cuda").to(torch.int32)
        cache = ops.Cache(0, Hk, rows, (n(B, case["appended"], Hk, D), n(B, case["appended"], Hk, D)))
    return dict(q=q, k=k, v=v, opts=ops.Attn(keys=keys, cache=cache))


def _prepare_linear(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    n = lambda s, *shape: (torch.randn(*shape, generator=g, device="cuda") * s).to(dt)
    m, nn, k = case["m"], case["n"], case["k"]
    wide = 2 * nn if case["gated"] else nn
    act = {"none": ops.Act.NONE, "gelu": ops.Act.GELU, "gelu_tanh": ops.Act.GELU_TANH, "silu": ops.Act.SILU}[case["act"]]
    return dict(x=n(1.0, m, k), w=n(0.02, wide, k),
                opts=ops.Linear(bias=n(0.02, wide) if case["bias"] else None, act=act, gated=case["gated"],
                                residual=n(1.0, m, nn) if case["residual"] else None))


def prepare(case, seed):
    if "model" in case:
        state = _prepare_model(case, seed)
    elif case["path"] == "linear":
        state = _prepare_linear(case, seed)
    else:
        state = _prepare_attention(case, seed)
    state["path"] = case["path"]
    return state


def run(state):
    path = state["path"]
    if path == "heads":
        return state["plans"].run(state["texts"])
    if path == "packed":
        return np.stack(state["embedder"].embed(state["texts"]))
    if path == "native":
        return state["runner"].run(state["ids"], state["aux"], state["out"])
    if path == "plan":
        state["plan"].run(state["ids"], state["aux"], state["out"])
        state["plan"].stream.synchronize()  # the rows are read on the host
        return state["out"]
    if path == "linear":
        return ops.linear(state["x"], state["w"], state["opts"])
    return ops.attention(state["q"], state["k"], state["v"], state["opts"])


# ---------------------------------------------------------------------------------- accounting
def _stack_work(model, lens):
    """Parameters read once, and the operations of the real tokens: 2 per weight and
    token, 4 * head width per visible (query, key) pair and query head."""
    c = STACKS[model][0]()
    D, tokens = c.hidden_size, sum(lens)
    if model == "xlmr":
        layers, per_layer, width = c.num_hidden_layers, 4 * D * D + 2 * D * c.intermediate_size, D
        pairs = layers * sum(n * n for n in lens)
    elif model == "qwen3":
        width, kv = c.num_attention_heads * c.head_dim, c.num_key_value_heads * c.head_dim
        layers, per_layer = c.num_hidden_layers, D * (width + 2 * kv) + width * D + 3 * D * c.intermediate_size
        pairs = layers * sum(n * (n + 1) // 2 for n in lens)
    else:
        layers, per_layer, width = c.num_hidden_layers, 4 * D * D + 3 * D * c.intermediate_size, D
        wide = -(-layers // c.global_attn_every_n_layers)
        half = c.local_attention // 2
        near = sum(min(i + half, n - 1) - max(i - half, 0) + 1 for n in lens for i in range(n))
        pairs = wide * sum(n * n for n in lens) + (layers - wide) * near
    return {"bytes": 2 * layers * per_layer + tokens * (2 * D + 4) + 4 * len(lens) * D,
            "flops": 2 * layers * per_layer * tokens + 4 * width * pairs}


def work(case):
    if "model" in case:
        return _stack_work(case["model"], _lengths(case.get("rows") or case["texts"], case["shortest"], case["longest"]))
    size = 4 if case["dtype"] == "float32" else 2
    if case["path"] == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        wide = 2 * n if case["gated"] else n
        extra = (wide if case["bias"] else 0) + (m * n if case["residual"] else 0)
        return {"bytes": size * (m * k + wide * k + m * n + extra), "flops": 2 * m * wide * k}
    B, T, H, Hk, D = (case[k] for k in ("batch", "queries", "heads", "kv_heads", "head_dim"))
    keys = sum(_lengths(B, case["shortest"], case["cache"])) + B * case.get("appended", 0)
    return {"bytes": size * (2 * keys * Hk * D + 2 * B * T * H * D), "flops": 4 * T * keys * H * D}


def tolerance(case):
    # A stack chains eight 16-bit roundings a layer: two correct implementations of the
    # 28-layer bf16 one differ by 1.2e-2 in its hidden states, of the 22-layer bf16 one
    # by 8e-3, of the 24-layer f16 one by 1.2e-3.
    if "model" in case:
        return {"rel": {"xlmr": 4e-3, "modernbert": 1.2e-2, "qwen3": 1.5e-2}[case["model"]]}
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 1e-2 if case["dtype"] == "bfloat16" else 2e-3}
