"""The training kernel's bounded waits: run with no MMA issued, its groups give
up, a whole warp at a time where warp-wide operations follow, and it returns
without adding to the gradients."""
import numpy as np
import pytest

import atlas_rt
from test_rc_gpu import HI, LO, random_records, scaled_params

pytestmark = pytest.mark.gpu


def test_training_goes_on_after_waits_that_gave_up():
    import torch
    ctx = atlas_rt.Context(device=0)
    rc = atlas_rt.RadianceCache(ctx, LO, HI, log2_table=14, seed=3)
    try:
        params = scaled_params(rc, 8)
        q = torch.from_numpy(random_records(700, 9)).cuda()
        rc.set_params(*params)
        first = rc.train_batch(q)           # leaves the gradients at zero, and says so
        trained = rc.get_params()
        assert rc.selftest_wait_timeout()   # the inference kernel's waits and the training kernel's
        for a, b in zip(trained, rc.get_params()):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        second = rc.train_batch(q)
        rc.set_params(*params)
        assert np.isclose(rc.train_batch(q), first, rtol=1e-3)
        assert np.isclose(rc.train_batch(q), second, rtol=1e-3)
    finally:
        rc.close()
        ctx.close()
