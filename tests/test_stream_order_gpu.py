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


def _late(copies):
    """Queues the copies behind about 50 ms of other work of torch's current stream."""
    import torch
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)
    for dst, src in copies:
        dst.copy_(src)


def test_passes_wait_for_data_and_outputs(ertm, orc):
    """Data, images, traces, perturbations, residuals and gradients that torch is still filling
    or clearing: the results are those of host arrays."""
    import torch
    shape, pml = (60, 1, 80), (8, 8, 0, 0, 8, 8)
    src, rec = geometry(shape, pml)
    kw = dict(nx=80, ny=1, nz=60, dx=10, dy=10, dz=10, dt_ms=0.8, nt=60, pml=pml)
    shot = ertm.Shot(*src, wavelet=orc.ricker(25.0, 8e-4), **rec)
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    zeros = lambda s: torch.full(s, 7.0, device="cuda")

    def check(call, inputs, want):
        ins, outs = [cuda(a) for a in inputs], [zeros(w.shape) for w in want]
        filled = [cuda(a) * 0 - 3 for a in inputs]
        _late([(f, i) for f, i in zip(filled, ins)] + [(o, torch.zeros_like(o)) for o in outs])
        call(filled, outs)
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert np.array_equal(o.cpu().numpy(), w)

    with ertm.Context(ertm.Config(**kw)) as ctx:
        m = model(shape, seed=9)
        ctx.set_model(ertm.TRUE_MODEL, *m)
        ctx.set_model(ertm.MIGRATION_MODEL, *m)
        d = ctx.forward_together_using_real_model(shot)
        check(lambda i, o: ctx.forward_together_using_real_model(shot, out=o[0]), [], [d])
        img = ctx.rtm_shot(shot, d)
        check(lambda i, o: ctx.rtm_shot(shot, i[0], *o), [d], img)
    with ertm.Context(ertm.Config(**kw, boundary=ertm.BOUNDARY_SPONGE_CUBIC, sponge_coef=150.0)) as ctx:
        ctx.set_model(ertm.MIGRATION_MODEL, *m)
        r = [(0.05 * np.random.default_rng(q).standard_normal(shape)).astype(np.float32) for q in range(3)]
        d = ctx.born_forward_shots([shot, shot], *r)
        check(lambda i, o: ctx.born_forward_shots([shot, shot], *i, out=o[0]), r, [d])
        g = ctx.born_adjoint_shots([shot, shot], d)
        check(lambda i, o: ctx.born_adjoint_shots([shot, shot], i[0], *o), [d], g)
