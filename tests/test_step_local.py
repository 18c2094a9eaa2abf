"""The short way of a single token through local blocks: the same logits as the general code, and the general code where the short way does not apply."""
import threading

import pytest
import torch

from cake_b200.model import B200Transformer, Cache, Context, TextModelBase
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
