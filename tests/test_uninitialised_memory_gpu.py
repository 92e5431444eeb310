"""Results do not depend on what freshly allocated device memory held (GPU).

Nothing promises that cudaMalloc returns zeros (other processes' memory is scrubbed,
this process's own need not be).  The same calls run in two child processes, one of
them with a preloaded cudaMalloc that fills every allocation with 0xff (NaN as
floats); the outputs are the same bits."""
import os
import shutil
import subprocess
import sys
import textwrap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int cudaMalloc(void **p, size_t n)
{
    void *h = dlopen("libcudart.so.12", RTLD_NOLOAD | RTLD_LAZY);
    if (!h) return 999;
    int rc = ((int (*)(void **, size_t))dlsym(h, "cudaMalloc"))(p, n);
    if (!rc && n) rc = ((int (*)(void *, int, size_t))dlsym(h, "cudaMemset"))(*p, 0xff, n);
    if (!rc) rc = ((int (*)(void))dlsym(h, "cudaDeviceSynchronize"))();
    return rc;
}
"""

CHILD = textwrap.dedent("""
    import importlib, sys
    import numpy as np
    sys.path[:0] = [{repo!r}, {tests!r}]
    ertm = importlib.import_module("2d_and_3d_elastic_reverse_time_migration_b200")
    from _cases import model
    rng = np.random.default_rng(3)
    out = {{}}

    def context(shape, pml, nt, **kw):
        nz, ny, nx = shape
        ctx = ertm.Context(ertm.Config(nx=nx, ny=ny, nz=nz, dx=10, dy=10, dz=10, dt_ms=0.8, nt=nt, pml=pml, **kw))
        ctx.set_model(ertm.MIGRATION_MODEL, *model(shape))
        ctx.set_model(ertm.TRUE_MODEL, *model(shape, seed=8))
        return ctx

    w = np.sin(np.arange(24) / 3.0).astype(np.float32)
    # sources beside the edge, so that every edge cell is reached
    for every, nm in ((0, 0), (20, 0), (20, 3)):
        visco = dict(visco_nmech=nm, visco_qp=100.0, visco_qs=50.0, visco_f0=15.0) if nm else {{}}
        ctx = context((44, 1, 70), (6, 6, 0, 0, 6, 6), 64, boundary=ertm.BOUNDARY_SPONGE_CUBIC, sponge_coef=50.0,
                      checkpoint_every=every, **visco)
        shots = [ertm.Shot(sx, 0, 3, wavelet=w, rx0=1, nrx=68, rz=2) for sx in (3, 35, 66)]
        r = [(0.1 * rng.standard_normal((44, 1, 70))).astype(np.float32) for _ in range(3)]
        d = ctx.born_forward_shots(shots, *r)
        out[f"d{{every}}_{{nm}}"] = d
        for q, g in enumerate(ctx.born_adjoint_shots(shots, d)):
            out[f"g{{every}}_{{nm}}_{{q}}"] = g
    for name, shape, pml in (("2d", (60, 1, 90), (8, 8, 0, 0, 8, 8)), ("3d", (34, 30, 46), (6, 6, 6, 6, 6, 6))):
        for order, b, kw in ((8, ertm.BOUNDARY_CPML, {{}}), (12, ertm.BOUNDARY_SPONGE_COS, dict(sponge_coef=60.0))):
            ctx = context(shape, pml, 60, order=order, boundary=b, **kw)
            nz, ny, nx = shape
            shot = ertm.Shot(nx // 2, ny // 2, 9, wavelet=w, rx0=8, nrx=nx - 16, ry0=8 if ny > 1 else 0,
                             nry=ny - 16 if ny > 1 else 1, rz=9)
            if ny == 1:
                ctx.set_angles()
            d = ctx.forward_together_using_real_model(shot)
            out[f"d{{name}}{{order}}"] = d
            for q, g in enumerate(ctx.rtm_shot(shot, d)):
                out[f"i{{name}}{{order}}_{{q}}"] = g
            if ny == 1:
                out[f"a{{name}}{{order}}_0"], out[f"a{{name}}{{order}}_1"] = ctx.get_angles()
    np.savez(sys.argv[1], **out)
""")


def test_poisoned_allocations_change_nothing(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    assert cc, "needs a C compiler for the preloaded cudaMalloc"
    src, so = tmp_path / "poison.c", tmp_path / "poison.so"
    src.write_text(SHIM)
    subprocess.run([cc, "-shared", "-fPIC", "-O1", "-o", str(so), str(src), "-ldl"], check=True)
    tests = os.path.dirname(os.path.abspath(__file__))
    code = CHILD.format(repo=os.path.dirname(tests), tests=tests)
    got = []
    for name, extra in (("plain", {}), ("poisoned", {"LD_PRELOAD": str(so)})):
        path = str(tmp_path / f"{name}.npz")
        subprocess.run([sys.executable, "-c", code, path], check=True, env={**os.environ, **extra}, timeout=300)
        got.append(dict(np.load(path)))
    plain, poisoned = got
    bad = [k for k in plain if not np.array_equal(plain[k], poisoned[k], equal_nan=True)]
    assert all(np.isfinite(v).all() for k, v in plain.items() if k[0] in "dg")
    assert not bad, ", ".join(bad)
