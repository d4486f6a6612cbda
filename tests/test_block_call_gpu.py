"""A pre-norm block as one call of the kernel library: the bits and the launches of its parts run one by one."""
import numpy as np
import pytest
import torch

from bitwise_b200 import LlamaConfig, Model
from bitwise_b200.cache.storage import build_cache
from bitwise_b200.engine.step import StepEntry, Stepper
from bitwise_b200.parts.block import PreNormBlock

pytestmark = pytest.mark.gpu


def _steps(model, cfg, parts, monkeypatch, steps, pages=120, max_rows=400, max_seqs=24):
    """Logits of every row of the steps, and launches."""
    taken = []
    if parts:
        monkeypatch.setattr(PreNormBlock, "_in_one_call", lambda self, ctx, x, cache: False)
    else:
        whole = PreNormBlock._in_one_call
        monkeypatch.setattr(PreNormBlock, "_in_one_call", lambda self, ctx, x, cache: taken.append(whole(self, ctx, x, cache)) or taken[-1])
    manager, storage = build_cache(model.decoder, pages, 16, max_seqs, torch.bfloat16, model.device)
    st = Stepper(model.decoder, manager, storage, model.ops, max_rows=max_rows, max_seqs=max_seqs, max_tokens_per_request=max_rows + 240,
                 use_graphs=False)
    rng = np.random.default_rng(3)
    tok = lambda n: rng.integers(0, cfg.vocab_size, n).tolist()
    before, out = model.ops.launches, []
    for step in steps:
        out.append(st.run([StepEntry(r, tok(n), list(range(n))) for r, n in step]).clone())
    torch.cuda.synchronize()
    monkeypatch.undo()
    assert parts or (taken and all(taken)), "the call was not taken"
    return out, model.ops.launches - before


def _same(model, cfg, monkeypatch, steps, **sizes):
    one, one_launches = _steps(model, cfg, False, monkeypatch, steps, **sizes)
    parts, parts_launches = _steps(model, cfg, True, monkeypatch, steps, **sizes)
    for i, (a, b) in enumerate(zip(one, parts)):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32)), f"step {i}"
    assert one_launches == parts_launches
    assert not model.ops.device_failure()


@pytest.mark.parametrize("hidden,heads,kv_heads,head_dim,inter", [(192, 3, 1, 64, 256), (256, 4, 4, 64, 200), (256, 4, 1, 128, 512),
                                                                 (96, 6, 2, 16, 104), (1024, 16, 4, 64, 2048)])
def test_one_call_gives_the_bits_of_the_parts(hidden, heads, kv_heads, head_dim, inter, monkeypatch):
    cfg = LlamaConfig(vocab_size=320, hidden_size=hidden, num_hidden_layers=2, num_attention_heads=heads, num_key_value_heads=kv_heads,
                      head_dim=head_dim, intermediate_size=inter, rms_norm_eps=1e-5, tie_word_embeddings=True, max_position_embeddings=640)
    model = Model.random(cfg, seed=5, dtype="bfloat16", device="cuda:0", fast=True, std=0.05)
    # a prompt in portions, single rows, and both side by side
    _same(model, cfg, monkeypatch, [[("a", 300)], [("a", 1), ("b", 70), ("c", 1)], [("a", 1)], [("a", 1), ("b", 1)],
                                    [("d%d" % i, 1) for i in range(18)] + [("a", 1)], [("a", 1)] + [("d%d" % i, 1) for i in range(18)],
                                    [("c", 17), ("b", 130)]])


def test_one_call_gives_the_bits_of_the_parts_on_block_pairs_and_the_streaming_kernel(monkeypatch):
    """A portion whose q/k/v product rotates and stores its outputs itself, and a step whose rows x key/value heads go to the streaming
    decode kernel."""
    cfg = LlamaConfig(vocab_size=320, hidden_size=2048, num_hidden_layers=2, num_attention_heads=32, num_key_value_heads=32, head_dim=64,
                      intermediate_size=1024, rms_norm_eps=1e-5, tie_word_embeddings=True, max_position_embeddings=1280)
    model = Model.random(cfg, seed=6, dtype="bfloat16", device="cuda:0", fast=True, std=0.03)
    for rows in (1000, 1120):
        assert model.ops.fuses_rope(rows, 2048, 32, 32, 64)
    steps = [[("a", 1000)]] + [[("d%d" % (8 * k + i), 140) for i in range(8)] for k in range(8)] + [[("d%d" % i, 1) for i in range(64)]]
    _same(model, cfg, monkeypatch, steps, pages=64 + 64 * 10, max_rows=1120, max_seqs=65)


@pytest.mark.parametrize("what", ["cache type", "64-bit positions", "positions on the host", "rows' sequences on the host", "block table on the host",
                                  "tiles on the host"])
def test_what_the_call_does_not_take_goes_to_the_parts_and_their_checks(what):
    """(What the one call hands over without these checks is shown in test_block_call_cpu.py, where nothing reads it.)"""
    from bitwise_b200.kernels.ops import KernelError
    cfg = LlamaConfig(vocab_size=64, hidden_size=64, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=2, head_dim=16,
                      intermediate_size=64, tie_word_embeddings=True, max_position_embeddings=64)
    model = Model.random(cfg, seed=1, dtype="bfloat16", device="cuda:0", fast=True)
    manager, storage = build_cache(model.decoder, 8, 16, 2, torch.bfloat16, model.device)
    st = Stepper(model.decoder, manager, storage, model.ops, max_rows=32, max_seqs=2, max_tokens_per_request=64, use_graphs=False)
    ctx, _ = st.prepare([StepEntry("a", [1, 2, 3], [2])])
    view = ctx.cache_views[0]
    if what == "cache type":
        view.k = view.k.float()  # no cache of this precision
    elif what == "64-bit positions":
        ctx.pos = ctx.pos.long()
    elif what == "positions on the host":
        ctx.pos = ctx.pos.cpu()
    elif what == "rows' sequences on the host":
        ctx.row_seq = ctx.row_seq.cpu()
    elif what == "block table on the host":
        view.block_table = view.block_table.cpu()
    else:
        ctx.tile_sets = {h: (s, r0.cpu(), r, c) for h, (s, r0, r, c) in ctx.tile_sets.items()}
    with pytest.raises(KernelError):
        model.decoder.forward(ctx, ctx.cache_views)
