"""A model given as CUDA tensors is taken after the work that torch still has queued on them (GPU)."""
import numpy as np
import pytest

from _cases import geometry, model

pytestmark = pytest.mark.gpu


def test_set_model_waits_for_the_tensors(ertm, orc):
    import torch
    shape, pml = (60, 1, 80), (8, 8, 0, 0, 8, 8)
    m = model(shape, seed=9)
    src, rec = geometry(shape, pml)
    cfg = ertm.Config(nx=80, ny=1, nz=60, dx=10, dy=10, dz=10, dt_ms=0.8, nt=80, pml=pml)
    shot = ertm.Shot(*src, wavelet=orc.ricker(25.0, 8e-4), **rec)
    with ertm.Context(cfg) as ctx:
        ctx.set_model(ertm.TRUE_MODEL, *m)
        want = ctx.forward_together_using_real_model(shot)
    dev = [torch.full(shape, 3000.0, device="cuda") for _ in range(3)]
    src_t = [torch.from_numpy(a).cuda() for a in m]
    with ertm.Context(cfg) as ctx:
        ctx.set_model(ertm.TRUE_MODEL, *m)       # allocations made
        torch.cuda.synchronize()
        torch.cuda._sleep(100_000_000)           # about 50 ms before the model's values arrive
        for d, a in zip(dev, src_t):
            d.copy_(a)
        ctx.set_model(ertm.TRUE_MODEL, *dev)
        got = ctx.forward_together_using_real_model(shot)
    assert np.array_equal(got, want)
