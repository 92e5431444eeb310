"""A receiver pass on the 3D workload's own grid (GPU): 480 x 480 x 380 cells, C-PML.

test_config2_gpu.py holds modelling and the source pass on this grid to the FP64 oracle; here
it is the receiver pass: 30 reverse steps of injected data, all thirteen wavefields of the
P/S-split state.  At this size cell offsets are near their 32-bit range and every column
has 12 z chunks.  Receivers start 8 cells inside the x-minimum layer, so that the field is in
the slabs from the first step on.  Tolerance: that of the wavefields there, flat relative
L2 1e-5."""
import numpy as np
import pytest

from _cases import rel

pytestmark = pytest.mark.gpu

NT = 30


def test_receiver_pass_wavefields(ertm, orc, synth):
    with open("/proc/meminfo") as f:
        gb = next(int(l.split()[1]) for l in f if l.startswith("MemAvailable:")) / 1e6
    if gb < 48:
        pytest.skip(f"needs ~48 GB of free host memory for the FP64 oracle, {gb:.0f} GB free")
    wl = synth.layered_3d(smooth_sigma=0)
    nz, ny, nx = wl.shape
    assert (nz, ny, nx) == (380, 480, 480)
    p = wl.pml
    rec = dict(rx0=p - 8, nrx=(nx - 2 * p) // 3, drx=3, ry0=p, nry=(ny - 2 * p) // 5, dry=5, rz=p + 2)
    nrec = rec["nrx"] * rec["nry"]
    t = np.arange(NT)[:, None] / 6.0
    ph = np.random.default_rng(4).uniform(0, 6.28, nrec)
    data = np.stack([np.sin(t + ph + q) for q in range(3)]).astype(np.float32)
    w = orc.ricker(25.0, wl.dt_ms / 1000.0)
    src = (p + 8, p + 8, p + 8)
    g = orc.make_grid(nx, ny, nz, wl.dx, wl.dy, wl.dz, wl.dt_ms, R=4, boundary=orc.CPML, pml=(p,) * 6,
                      pml_r=1e-3, pml_f0=10.0, pml_vmax=float(wl.vp.max()))
    ref = orc.run_pass(g, wl.vp, wl.vs, wl.rho, orc.make_shot(*src, w, **rec), orc.RECEIVER, NT, data=data,
                       ex=orc.ExcitationArrays(wl.shape), want_fields=True)["fields"]
    cfg = ertm.Config(nx=nx, ny=ny, nz=nz, dx=wl.dx, dy=wl.dy, dz=wl.dz, dt_ms=wl.dt_ms, nt=NT, src_steps=2,
                      order=8, boundary=ertm.BOUNDARY_CPML, pml=(p,) * 6, pml_r=1e-3, pml_f0=10.0)
    shot = ertm.Shot(*src, wavelet=w, **rec)
    with ertm.Context(cfg) as ctx:
        ctx.set_model(ertm.MIGRATION_MODEL, wl.vp, wl.vs, wl.rho)
        ctx.forward_together_using_smoothed_model(shot)
        ctx.backward_together_using_smoothed_model(shot, data)
        bad = {}
        for name in ref:
            e = rel(ctx.get_wavefield(name), ref[name])
            assert np.any(ref[name]), name
            if not e <= 1e-5:
                bad[name] = e
    assert not bad, bad
