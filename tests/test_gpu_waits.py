"""The bounded waits of the tensor-core kernels (mbar_wait_lim): a wait that nothing ends gives up after its limit, sets the error word that
the next synchronising call reports, and the thread's later waits return at once.  Nothing faults: the probe kernel waits on a
barrier of its own, returns, and the context stays usable."""
import ctypes

import numpy as np
import pytest

from cake_b200.capi import CakeB200Error, check, lib
from cake_b200.model import B200Transformer, Context
from tests.util import checkpoint, medium_config, rand_x, to_np

pytestmark = pytest.mark.gpu


def probe(ctx, arrivals, tries, ok, kcycles):
    fn = lib().cake_b200_debug_wait
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_uint32, ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_int)]
    check(fn(ctx.h, arrivals, tries, ok, kcycles))


def test_a_wait_that_runs_out_is_reported_and_the_thread_does_not_wait_again():
    cfg = medium_config()
    ctx = Context(cfg, checkpoint(cfg, "bf16", seed=3), "bf16")
    ok, kcycles = (ctypes.c_int * 2)(), (ctypes.c_int * 2)()
    try:
        probe(ctx, 2, 256, ok, kcycles)      # both arrivals came: no error
        assert list(ok) == [1, 1]
        ctx.sync()
        probe(ctx, 1, 8192, ok, kcycles)     # one of two: the first wait takes all of its tries, the second one at most two
        print(f"8192 tries {kcycles[0]} kcycles, then {kcycles[1]}")
        assert list(ok) == [0, 0] and kcycles[0] < 2000000 and kcycles[1] < kcycles[0] / 100
        with pytest.raises(CakeB200Error, match="gave up a wait"):
            ctx.sync()
        blk = B200Transformer.load(cfg.layer_name(0), ctx)
        ctx.cache.clear()
        x = ctx.to_device(rand_x((1, 40, cfg.hidden_size), "bf16", seed=1))
        y = blk.forward(x, 0, 0, ctx)
        ctx.sync()
        assert np.isfinite(to_np(y)).all()
    finally:
        ctx.close()
