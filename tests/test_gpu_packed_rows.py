"""Packed rows: a padded batch computed without its trailing padding gives the pooled rows
of the padded batch. Sizes sit where the layout can go wrong: rows that end on, before and
behind a 64-position block, rows of one token and of none, masks with holes, lengths that
are no multiple of the block, batches through the few-tile, one-CTA and CTA-pair GEMMs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STACKS = ["xlmr", "qwen3", "modernbert"]


def _model(kind, hidden=512):
    from svod_b200 import encoders as E
    if kind == "xlmr":
        cfg = E.XlmRobertaConfig(vocab_size=500, hidden_size=hidden, num_hidden_layers=2, num_attention_heads=hidden // 64,
                                 intermediate_size=2 * hidden, max_position_embeddings=1100)
        return E.XlmRobertaEncoder.random_init(cfg, seed=3)
    if kind == "qwen3":
        cfg = E.Qwen3Config(vocab_size=500, hidden_size=hidden, num_hidden_layers=2, num_attention_heads=hidden // 128,
                            num_key_value_heads=hidden // 256, intermediate_size=2 * hidden)
        return E.Qwen3Embedder.random_init(cfg, seed=4)
    cfg = E.ModernBertConfig(vocab_size=500, hidden_size=hidden, num_hidden_layers=4, num_attention_heads=hidden // 64,
                             intermediate_size=hidden)
    return E.ModernBertEncoder.random_init(cfg, seed=5)


def _batch(lens, L, kind, holes=False, seed=0):
    r = np.random.RandomState(seed)
    ids = torch.full((len(lens), L), 1, dtype=torch.int32)
    mask = torch.zeros(len(lens), L, dtype=torch.bool)
    for i, n in enumerate(lens):
        ids[i, :n] = torch.from_numpy(r.randint(5, 500, n).astype(np.int32))
        mask[i, :n] = True
        if holes and n > 8:
            mask[i, torch.from_numpy(r.choice(n - 1, n // 5, replace=False))] = False
    aux = torch.tensor(lens, dtype=torch.int32) if kind == "qwen3" else mask
    return ids.cuda(), aux.cuda()


# (row lengths, L): few-tile / one-CTA / CTA-pair projections; L on and off the block
CASES = [
    ([130, 1, 64, 65, 63, 128, 200, 7], 200),
    ([384, 129, 128, 127], 384),
    ([301, 33, 97, 192, 1, 320], 321),
    ([1024, 700, 64, 1, 513, 960, 1000, 130], 1024),
    ([512] * 16, 512),
]


def _close(got, want, kind):
    # the same values bit for bit up to the pooling, whose f32 mean of up to 1024 tokens may be summed in
    # another order: 1024 * 2^-24 (a key block missing from one row of a batch is 1e-2 of that row)
    tol = 1024 * 2.0 ** -24
    got, want = got.double().cpu(), want.double().cpu()
    assert torch.isfinite(got).all()
    assert (got - want).norm() <= tol * want.norm()
    assert ((got - want).norm(dim=1) <= tol * want.norm(dim=1).clamp_min(1e-30)).all()


@pytest.mark.parametrize("kind", STACKS)
@pytest.mark.parametrize("case", range(len(CASES)))
def test_matches_the_padded_batch(kind, case, monkeypatch):
    from svod_b200 import ops
    lens, L = CASES[case]
    model = _model(kind)
    ids, aux = _batch(lens, L, kind, seed=case)
    assert ops.rows_pay(*ids.shape)
    got = model.forward(ids, aux)
    assert ops._packed.length is None
    ops.device_status()
    monkeypatch.setattr(ops, "rows_pay", lambda b, n: False)
    _close(got, model.forward(ids, aux), kind)


@pytest.mark.parametrize("kind,pooling", [("xlmr", "cls"), ("xlmr", "mean"), ("modernbert", "mean"), ("modernbert", "cls")])
@pytest.mark.parametrize("dtype", [torch.bool, torch.int64])
def test_masks_with_holes_and_empty_rows(kind, pooling, dtype, monkeypatch):
    from svod_b200 import ops
    model = _model(kind)
    model.cfg.pooling = pooling
    ids, mask = _batch([150, 0, 320, 65, 0], 320, kind, holes=True)
    mask[3, :] = False
    mask[3, 40:60] = True  # hidden tokens before and behind
    mask = mask.to(dtype)
    got = model.forward(ids, mask)
    monkeypatch.setattr(ops, "rows_pay", lambda b, n: False)
    want = model.forward(ids, mask)
    live = [0, 2, 3] if pooling == "mean" else range(5)  # the mean of no token is zero on both sides
    _close(got[list(live)], want[list(live)], kind)
    assert (got[1] == want[1]).all() or pooling == "cls"


@pytest.mark.parametrize("pooling", ["cls", "mean"])
@pytest.mark.parametrize("value", [0.5, 1 << 32])
def test_masks_of_another_type_attend_where_they_are_nonzero(value, pooling, monkeypatch):
    from svod_b200 import ops
    model = _model("modernbert")
    model.cfg.pooling = pooling
    ids, mask = _batch([300, 129, 64, 200], 300, "modernbert")
    aux = mask.to(torch.float32 if value < 1 else torch.int64)
    aux[:, 20:60] *= value  # an integer conversion would leave 0 of it
    got = model.forward(ids, aux)
    monkeypatch.setattr(ops, "rows_pay", lambda b, n: False)
    # (the pooling of a padded batch converts to i32, so the mean of the int64 case has no reference there)
    _close(got, model.forward(ids, mask if value > 1 else aux), "modernbert")


def test_lengths_outside_the_row(monkeypatch):
    from svod_b200 import ops
    model = _model("qwen3")
    ids, _ = _batch([300] * 4, 300, "qwen3")
    aux = torch.tensor([-3, 0, 1000, 77], dtype=torch.int32).cuda()
    got = model.forward(ids, aux)
    monkeypatch.setattr(ops, "rows_pay", lambda b, n: False)
    _close(got, model.forward(ids, aux), "qwen3")


@pytest.mark.parametrize("kind", STACKS)
def test_plan_replays_serve_other_lengths(kind, monkeypatch):
    """One captured plan, batches of other lengths one after the other: nothing of the one
    before shows, on the Python plan and the native one (whose L is off the block)."""
    from svod_b200 import encoders as E
    from svod_b200 import native, ops
    model = _model(kind)
    B, L = 6, 300
    plan = E.Plan(model, B, L, "lengths" if kind == "qwen3" else "mask").capture()
    run = {"xlmr": native.NativeXlmRoberta, "qwen3": native.NativeQwen3, "modernbert": native.NativeModernBert}[kind](model)
    for seed, lens in enumerate([[300] * 6, [1, 2, 64, 65, 300, 128], [5] * 6, [256, 257, 255, 1, 300, 64]]):
        ids, aux = _batch(lens, L, kind, seed=seed)
        out = torch.empty(B, model.cfg.hidden_size).pin_memory()
        plan.run(ids.cpu().pin_memory(), aux.cpu().pin_memory(), out)
        plan.check()
        nat = run.run(ids.cpu().numpy(), aux.cpu().numpy().astype(run.aux_dtype))
        with monkeypatch.context() as m:
            m.setattr(ops, "rows_pay", lambda b, n: False)
            want = model.forward(ids, aux)
        _close(out, want, kind)
        assert (nat == out.numpy()).all()


def test_calls_without_a_kernel_fall_back():
    """A stack whose rows the fused kernels do not take runs padded, and says nothing."""
    from svod_b200 import encoders as E
    from svod_b200 import ops
    cfg = E.ModernBertConfig(vocab_size=500, hidden_size=320, num_hidden_layers=2, num_attention_heads=10,
                             intermediate_size=320)  # 32-wide heads: the rotation runs outside the store
    model = E.ModernBertEncoder.random_init(cfg, seed=1)
    ids, mask = _batch([200, 100, 256, 33], 256, "modernbert")
    got = model.forward(ids, mask)
    assert ops._packed.length is None
    want = ops.pool(model.hidden(ids, mask), mask, ops.POOL_MEAN)
    _close(got, want, "modernbert")
    with pytest.raises(ops.OpsError) as e:
        with ops.PackedRows(mask, 256):
            ops.heads(torch.empty(4, 256, 960, dtype=torch.bfloat16, device="cuda"), ops.Qkv(10, 10, 32))
    assert e.value.code == ops.ERR_UNSUPPORTED
    assert ops._packed.length is None


@pytest.mark.parametrize("hidden,heads,off", [(384, 12, ""), (2304, 18, ""), (512, 8, "out"), (512, 8, "weight")])
def test_a_stack_without_kernels_for_it_runs_once(hidden, heads, off, monkeypatch):
    """Widths the fused pooling does not take and a result off the 16-byte grid (nothing of the
    packed stack is launched), and a final norm's weight off it, which only the last op sees (the
    second run knows): launches of an eager run and of a captured plan."""
    from svod_b200 import encoders as E
    from svod_b200 import native, ops
    kind = "modernbert" if off == "weight" else "xlmr"
    if kind == "xlmr":
        cfg = E.XlmRobertaConfig(vocab_size=500, hidden_size=hidden, num_hidden_layers=2, num_attention_heads=heads,
                                 intermediate_size=512, max_position_embeddings=300)
        model = E.XlmRobertaEncoder.random_init(cfg, seed=2)
    else:
        model = _model(kind, hidden)
        model.p["final_ln_w"] = torch.ones(hidden + 1, dtype=model.cfg.dtype, device="cuda")[1:]
    ids, mask = _batch([200, 100, 256, 33], 256, kind)
    out = torch.empty(4 * hidden + 1, device="cuda")[1:].view(4, hidden) if off == "out" else None

    def launches(call):
        before = ops.launches
        call()
        return ops.launches - before

    with monkeypatch.context() as m:
        m.setattr(ops, "rows_pay", lambda b, n: False)
        want = model.forward(ids, mask).clone()
        once = launches(lambda: model.forward(ids, mask, out))
    assert ops.rows_pay(*ids.shape)
    first = launches(lambda: model.forward(ids, mask, out))
    assert first > once if off == "weight" else first == once
    assert launches(lambda: model.forward(ids, mask, out)) == once
    plan = E.Plan(model, 4, 256, "mask", out=out if out is not None else torch.empty(4, hidden, device="cuda"))
    assert launches(plan.capture) == 2 * once  # the eager run and the captured one
    host_out = torch.empty(4, hidden).pin_memory()
    plan.run(ids.cpu().pin_memory(), mask.cpu().pin_memory(), host_out)
    plan.check()
    _close(host_out, want, kind)
    got = (native.NativeXlmRoberta if kind == "xlmr" else native.NativeModernBert)(model).run(ids.cpu().numpy(), mask.cpu().numpy().astype(np.uint8))
    _close(torch.from_numpy(got), want, kind)
