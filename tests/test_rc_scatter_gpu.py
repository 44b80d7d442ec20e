"""The training kernel's gradient scatter, which sums runs of neighbouring
records in one grid cell before it adds them, and its direct output into the
caller's device buffers: against the warp-level kernel, which adds every
record on its own.  Both round the same values to BF16 and differ in the order
of FP32 additions and in rare BF16 roundings of the deltas, so the gradient
vectors are compared at 1 % relative L2, as the two kernels always are."""
import numpy as np
import pytest

import atlas_rt
from test_rc_gpu import HI, LO, random_records, rel, scaled_params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def caches():
    ctx = atlas_rt.Context(device=0)
    tc = atlas_rt.RadianceCache(ctx, LO, HI, log2_table=14, seed=3)
    warp = atlas_rt.RadianceCache(ctx, LO, HI, log2_table=14, seed=3, warp_mma_training=True)
    params = scaled_params(tc, 1)       # once: it scales what the cache holds
    for rc in (tc, warp):
        rc.set_params(*params)
    yield ctx, tc, warp
    tc.close()
    warp.close()
    ctx.close()


def records(n, run, seed):
    """Runs of `run` records at one position (0: all at one, 1: all apart)."""
    rec = random_records(n, seed)
    if run != 1:
        first = np.zeros(n, int) if run == 0 else np.arange(n) // run * run
        rec[:, 0:3] = rec[first, 0:3]
    return rec


@pytest.mark.parametrize("n", [1, 31, 128, 129, 700])
@pytest.mark.parametrize("run", [0, 1, 2, 3, 9, 32, 33])
def test_scatter_of_runs(caches, n, run):
    import torch
    _, tc, warp = caches
    q = torch.from_numpy(records(n, run, n + 7 * run)).cuda()
    got = [torch.full((k,), 3.0, device="cuda") for k in (tc.n_mlp, tc.n_grid)]     # cleared by the call
    loss = tc.gradients(q, *got)
    want = [np.zeros(k, np.float32) for k in (warp.n_mlp, warp.n_grid)]
    wloss = warp.gradients(q, *want)
    assert abs(loss - wloss) <= 1e-3 * abs(wloss)
    for g, w in zip(got, want):
        assert rel(g.cpu().numpy(), w) < 0.01
    # the same through the cache's own buffers (host memory; an unaligned device buffer)
    host = [np.zeros(k, np.float32) for k in (tc.n_mlp, tc.n_grid)]
    tc.gradients(q, *host)
    odd = torch.zeros(tc.n_grid + 1, device="cuda")
    tc.gradients(q, host[0], odd[1:])
    for g, h in zip(got, host):
        assert rel(g.cpu().numpy(), h) < 1e-5
    assert rel(odd[1:].cpu().numpy(), host[1]) < 1e-5 and float(odd[0]) == 0.0


def test_training_after_direct_gradients_starts_from_zero(caches):
    """Gradients written into the caller's buffers leave the cache's own as
    they were: a training step before and one after agree with two in a row."""
    import torch
    ctx, tc, _ = caches
    q = torch.from_numpy(random_records(600, 5)).cuda()
    losses, params = [], scaled_params(tc, 2)
    for between in (False, True):
        tc.set_params(*params)
        a = tc.train_batch(q)
        if between:
            tc.gradients(q, torch.zeros(tc.n_mlp, device="cuda"), torch.zeros(tc.n_grid, device="cuda"))
        losses.append((a, tc.train_batch(q)))
    assert np.allclose(losses[0], losses[1], rtol=1e-3)
