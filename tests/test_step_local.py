"""The short way of a single token through local blocks: the same logits as the general code, and the general code where the short way does not apply."""
import threading

import pytest
import torch

from cake_b200.model import B200Transformer, Cache, Context, TextModelBase
from tests.cpu_ctx import CpuContext, use_emulation
from tests.util import checkpoint, medium_config


class Elsewhere(B200Transformer):
    """A block whose forward_batch is its own."""
    calls = 0

    def forward_batch(self, x, batch, ctx, blocks=None):
        Elsewhere.calls += 1
        return super().forward_batch(x, batch, ctx, blocks=blocks)


@pytest.fixture
def model():
    cfg = medium_config()
    ctx = Context(cfg, checkpoint(cfg, "bf16", seed=3), "bf16")
    ctx.cache = Cache(ctx, 1, 64)
    yield TextModelBase.load(ctx)
    ctx.close()


def steps(m, toks, general):
    m.ctx.cache.clear()
    out = []
    for i, t in enumerate(toks):
        # a tuple is the general code's: only lists of one int take the short way
        with torch.cuda.stream(m.ctx.torch_stream):   # the stream that the logits are written on
            out.append(m.forward([(t,)] if general else [[t]], i).clone())
    m.ctx.sync()
    return torch.cat(out)


@pytest.mark.gpu
def test_short_way_gives_the_same(model):
    toks = [3, 17, 5, 9, 200]
    want = steps(model, toks, True)
    assert torch.equal(steps(model, toks, False), want) and model._run[0] == [b.h.value for b in model.blocks]
    assert torch.equal(steps(model, toks, False), want)
    for bad in (-1, 1 << 32, model.ctx.config.vocab_size):   # out of range: refused as before
        with pytest.raises(Exception):
            model.forward([[bad]], len(toks))


@pytest.mark.gpu
def test_blocks_of_another_make_are_asked(model):
    toks = [3, 17, 5]
    want = steps(model, toks, False)
    model.blocks[0].__class__ = Elsewhere   # (a run of blocks of one place is the first one's call)
    assert model._local_run() is None
    Elsewhere.calls = 0
    assert torch.equal(steps(model, toks, False), want) and Elsewhere.calls == len(toks)


@pytest.mark.gpu
def test_threads_have_rows_of_their_own(model):
    rows = {}

    def one(name):
        model.ctx.cache.clear()
        model.forward([[5]], 0)
        rows[name] = (model._step_rows.x, model._step_rows.y)
    one("here")
    t = threading.Thread(target=one, args=("there",))
    t.start()
    t.join()
    model.ctx.sync()
    assert len({r.data_ptr() for pair in rows.values() for r in pair}) == 4


@pytest.mark.parametrize("where", ["nowhere", "a block", "its class", "the base class", "a block's place", "a block's name"])
def test_who_asks_a_block_is_not_passed_by(where, monkeypatch, tmp_path):
    """A tracer on one block, on all blocks of a make, on where they say they live or what they are called: asked for the prompt, and for every token behind it."""
    use_emulation(monkeypatch, tmp_path)
    cfg = medium_config()
    ctx = CpuContext(cfg, checkpoint(cfg, "bf16", seed=3), "bf16")
    try:
        m = TextModelBase.load(ctx)
        asked = []

        def traced(method):
            def call(*args, **kw):
                asked.append(method.__name__)
                return method(*args, **kw)
            return call

        class Own(B200Transformer):
            forward_batch = traced(B200Transformer.forward_batch)

        first = m.blocks[0]
        if where == "a block":
            first.forward_batch = traced(first.forward_batch)
        elif where == "its class":
            first.__class__ = Own
        elif where == "the base class":
            monkeypatch.setattr(B200Transformer, "forward_batch", traced(B200Transformer.forward_batch))
        elif where == "a block's place":
            first.ident = traced(first.ident)
        elif where == "a block's name":
            first.layer_name = traced(first.layer_name)
        assert (m._local_run() is None) == (where != "nowhere")
        m.forward([[3, 5, 7]], 0)
        per_call = len(asked)
        assert bool(per_call) == (where != "nowhere")
        for i in range(2):
            m.forward([[9 + i]], 3 + i)
        assert len(asked) == 3 * per_call
    finally:
        ctx.close()
