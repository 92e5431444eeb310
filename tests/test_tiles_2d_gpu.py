"""The 2D step kernels and the Born kernels at the edges of their tiles, against the
oracle (GPU).  A CTA takes 64 columns and 4, 8 or 16 rows, the most rows that still give
one CTA per SM; the sizes here end exactly on a tile or one cell past it, for each number
of rows.  Tolerance: that of the parity tests, max(1e-5, 3 x the FP32 oracle's own
relative L2 error against FP64)."""
import numpy as np
import pytest

from _born_case import VISCO, born_case
from _cases import CPML, DT_MS, DX, SPONGE_CUBIC, geometry, model, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,nx,R,boundary", [
    (36, 64, 4, CPML), (37, 65, 6, SPONGE_CUBIC), (41, 129, 4, SPONGE_CUBIC), (43, 63, 6, CPML),   # 4 rows
    (296, 256, 4, CPML), (297, 257, 6, CPML), (303, 255, 4, SPONGE_CUBIC),                        # 8 rows
    (240, 640, 4, CPML), (241, 641, 6, SPONGE_CUBIC), (255, 639, 6, CPML)])                       # 16 rows
def test_2d_tiles_match_oracle(ertm, orc, nz, nx, R, boundary):
    shape, pml, nt = (nz, 1, nx), (11, 10, 0, 0, 9, 12), 150
    vp, vs, rho = model(shape, seed=5)
    g = orc.make_grid(nx, 1, nz, DX, DX, DX, DT_MS, R=R, boundary=boundary, pml=pml, pml_r=1e-3, pml_f0=10.0,
                      pml_vmax=float(vp.max()), sponge_coef=200.0)
    src, rec = geometry(shape, pml)
    src = (nx - pml[1] - 2, 0, nz - pml[5] - 4)           # in the last tiles of both axes
    rec["rz"] = nz - pml[5] - 2
    w = orc.ricker(25.0, DT_MS / 1000.0)
    oshot = orc.make_shot(*src, w, **rec)
    cfg = ertm.Config(nx=nx, ny=1, nz=nz, dx=DX, dy=DX, dz=DX, dt_ms=DT_MS, nt=nt, order=2 * R,
                      boundary=boundary, pml=pml, pml_r=1e-3, pml_f0=10.0, sponge_coef=200.0)
    with ertm.Context(cfg) as ctx:
        ctx.set_model(ertm.TRUE_MODEL, vp, vs, rho)
        shot = ertm.Shot(*src, wavelet=w, **rec)
        data = ctx.forward_together_using_real_model(shot)
        ctx.propagate(ertm.TRUE_MODEL, shot, nt)
        fields = {k: ctx.get_wavefield(k) for k in ("vx", "vz", "txx", "tzz", "txz")}
    ref, r32 = (orc.run_pass(g, vp, vs, rho, oshot, orc.MODEL, nt, want_fields=True, bits=b) for b in (64, 32))
    for k, f in fields.items():
        assert rel(f, ref["fields"][k]) <= max(1e-5, 3 * rel(r32["fields"][k], ref["fields"][k])), k
    for q in (0, 2):
        assert rel(data[q], ref["data"][q]) <= max(1e-5, 3 * rel(r32["data"][q], ref["data"][q])), q


# columns: 8 cells of left halo + nx over tiles of 64
@pytest.mark.parametrize("nz,nx,R,visco", [
    (44, 56, 4, False), (45, 57, 6, True),                # 4 rows
    (392, 184, 4, False), (393, 185, 6, True),            # 8 rows
    (336, 376, 6, False), (337, 377, 4, False)])          # 16 rows (elastic only)
def test_born_tiles_match_oracle(ertm, orc, nz, nx, R, visco):
    c = born_case(orc, nz=nz, nx=nx, nt=130, R=R)
    v = {}
    if visco:
        c["g"].visco_nmech, c["g"].visco_qp, c["g"].visco_qs, c["g"].visco_f0 = VISCO
        v = dict(zip(("visco_nmech", "visco_qp", "visco_qs", "visco_f0"), VISCO))
    src, rec = (nx - 13, 0, nz - 14), dict(rx0=10, nrx=nx - 20, drx=1, rz=nz - 12)
    s = orc.make_shot(*src, c["w"], **rec)
    m = [(0.05 * c["rng"].standard_normal(c["shape"])).astype(np.float32) for _ in range(3)]
    args = (c["g"], c["vp"], c["vs"], c["rho"], s, c["nt"])
    ref, r32 = (orc.born_forward(*args, *m, bits=b) for b in (64, 32))
    cfg = ertm.Config(nx=nx, ny=1, nz=nz, dx=10, dy=10, dz=10, dt_ms=1.0, nt=c["nt"], order=2 * R,
                      boundary=SPONGE_CUBIC, pml=c["pml"], sponge_coef=150.0, checkpoint_every=50, **v)
    with ertm.Context(cfg) as ctx:
        ctx.set_model(ertm.MIGRATION_MODEL, c["vp"], c["vs"], c["rho"])
        shot = ertm.Shot(*src, wavelet=c["w"], **rec)
        d = ctx.born_forward(shot, *m)
        dh = c["rng"].standard_normal(ref.shape).astype(np.float32)
        dh[1] = 0
        g = ctx.born_adjoint(shot, dh)
    for q in (0, 2):
        assert rel(d[q], ref[q]) <= max(1e-5, 3 * rel(r32[q], ref[q])), q
    gref, g32 = (orc.born_adjoint(*args, dh, bits=b) for b in (64, 32))
    for a, b, f in zip(g, gref, g32):
        assert rel(a, b) <= max(1e-5, 3 * rel(f, b))


# segments of 40 (the first shorter) and 75 steps (two) against one of 150 that is never
# rebuilt, bit for bit; 8 shots pass 100,000 cells (earlier segments rebuilt on a second
# stream), 2 do not
@pytest.mark.parametrize("nshots", [2, 8])
def test_born_segments_do_not_change_the_gradient(ertm, orc, nshots):
    c = born_case(orc, nz=110, nx=130, nt=150)
    rec = c["geo"]["rec"]
    dh = c["rng"].standard_normal((nshots, 3, 150, rec["nrx"])).astype(np.float32)
    dh[:, 1] = 0
    shots = [ertm.Shot(int(x), 0, 12, wavelet=c["w"], **rec) for x in np.linspace(15, 114, nshots)]
    g = {}
    for every in (150, 75, 40):
        cfg = ertm.Config(nx=130, ny=1, nz=110, dx=10, dy=10, dz=10, dt_ms=1.0, nt=150, order=8,
                          boundary=SPONGE_CUBIC, pml=c["pml"], sponge_coef=150.0, checkpoint_every=every)
        with ertm.Context(cfg) as ctx:
            ctx.set_model(ertm.MIGRATION_MODEL, c["vp"], c["vs"], c["rho"])
            g[every] = [ctx.born_adjoint_shots(shots, dh) for _ in range(2)]
    for every in (75, 40):
        for run in g[every]:
            for a, b in zip(run, g[150][0]):
                assert np.any(b) and np.array_equal(a, b), every


# passes on either side of the lines between direct launches and graphs, and with one, two and
# four graphs' worth of steps ahead, record the same samples bit for bit
@pytest.mark.parametrize("nz,nx,steps", [(60, 90, (20, 63, 64, 199, 200, 201, 260)), (632, 632, (20, 40)),
                                         (633, 633, (16, 20, 40, 70))])
def test_time_loop_forms_agree(ertm, orc, nz, nx, steps):
    shape, pml = (nz, 1, nx), (9, 8, 0, 0, 8, 9)
    m = model(shape, seed=6)
    src, rec = geometry(shape, pml)
    got = {}
    for nt in steps:
        cfg = ertm.Config(nx=nx, ny=1, nz=nz, dx=DX, dy=DX, dz=DX, dt_ms=DT_MS, nt=nt, pml=pml)
        with ertm.Context(cfg) as ctx:
            ctx.set_model(ertm.TRUE_MODEL, *m)
            got[nt] = ctx.forward_together_using_real_model(
                ertm.Shot(*src, wavelet=orc.ricker(25.0, DT_MS / 1000.0), **rec))
    longest = got[max(steps)]
    assert np.any(longest)
    for nt, d in got.items():
        assert np.array_equal(d, longest[:, :nt]), nt
