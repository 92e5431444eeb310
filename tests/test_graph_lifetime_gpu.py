"""A pass's graph is destroyed only when its replays are known to be done (GPU).

A preloaded cudaGraphExecDestroy asks for an event behind the graph's last replay: the child
process below runs 2D and 3D passes, several shots in one launch, and a grid change, and no
graph may be destroyed before its event has passed.  Every graph that was made is destroyed
by the time its context is."""
import json
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static struct { void *graph, *event; } last[64];   /* event: behind the graph's last replay */
static int n, made, gone, busy;
static void *real(const char *f) { return dlsym(dlopen("libcudart.so.12", RTLD_NOLOAD | RTLD_LAZY), f); }
int cudaGraphLaunch(void *g, void *s)
{
    int q = 0, rc = ((int (*)(void *, void *))real("cudaGraphLaunch"))(g, s);
    while (q < n && last[q].graph != g) q++;
    if (q == n) {
        if (n == 64) return 999;
        if (((int (*)(void **))real("cudaEventCreate"))(&last[n].event)) return 999;
        last[n++].graph = g;
    }
    if (!rc) rc = ((int (*)(void *, void *))real("cudaEventRecord"))(last[q].event, s);
    return rc;
}
int cudaGraphInstantiate(void **e, void *g, unsigned long long f)
{
    made++;
    return ((int (*)(void **, void *, unsigned long long))real("cudaGraphInstantiate"))(e, g, f);
}
int cudaGraphExecDestroy(void *e)
{
    gone++;
    for (int q = 0; q < n; q++)
        if (last[q].graph == e) {
            if (((int (*)(void *))real("cudaEventQuery"))(last[q].event) == 600) busy++;   /* cudaErrorNotReady */
            ((int (*)(void *))real("cudaEventDestroy"))(last[q].event);
            last[q] = last[--n];
            break;
        }
    return ((int (*)(void *))real("cudaGraphExecDestroy"))(e);
}
void seen(int *v) { v[0] = made; v[1] = gone; v[2] = busy; }
"""

CHILD = textwrap.dedent("""
    import ctypes, importlib, json, sys
    import numpy as np
    sys.path[:0] = [{repo!r}, {tests!r}]
    ertm = importlib.import_module("2d_and_3d_elastic_reverse_time_migration_b200")
    from _cases import model
    w = np.sin(np.arange(24) / 3.0).astype(np.float32)

    def context(shape, pml, nt):
        nz, ny, nx = shape
        ctx = ertm.Context(ertm.Config(nx=nx, ny=ny, nz=nz, dx=10, dy=10, dz=10, dt_ms=0.8, nt=nt, pml=pml))
        for which in (ertm.TRUE_MODEL, ertm.MIGRATION_MODEL):
            ctx.set_model(which, *model(shape))
        return ctx

    def shot(shape):
        nz, ny, nx = shape
        return ertm.Shot(nx // 2, ny // 2, 9, wavelet=w, rx0=8, nrx=nx - 16, ry0=8 if ny > 1 else 0,
                         nry=ny - 16 if ny > 1 else 1, rz=9)

    for shape, pml in (((90, 1, 120), (8, 8, 0, 0, 8, 8)), ((34, 30, 46), (6, 6, 6, 6, 6, 6))):
        with context(shape, pml, 600) as ctx:
            for _ in range(3):
                ctx.rtm_shot(shot(shape), ctx.forward_together_using_real_model(shot(shape)))
            ctx.set_grid(shape[2] - 2, shape[1], 400, 300)
    shape, pml = (34, 30, 46), (6, 6, 6, 6, 6, 6)
    cs = [context(shape, pml, 300) for _ in range(2)]
    data = [np.zeros((3, 300, shot(shape).nrec), np.float32)] * 2
    for _ in range(2):
        ertm.rtm_multi(cs, [shot(shape)] * 2, data)
    for c in cs:
        c.close()
    v = (ctypes.c_int * 3)()
    ctypes.CDLL(sys.argv[1]).seen(v)
    print(json.dumps(list(v)))
""")


def test_no_graph_is_destroyed_in_flight(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    assert cc, "needs a C compiler for the preloaded calls"
    src, so = tmp_path / "graphs.c", tmp_path / "graphs.so"
    src.write_text(SHIM)
    subprocess.run([cc, "-shared", "-fPIC", "-O1", "-o", str(so), str(src), "-ldl"], check=True)
    tests = os.path.dirname(os.path.abspath(__file__))
    code = CHILD.format(repo=os.path.dirname(tests), tests=tests)
    out = subprocess.run([sys.executable, "-c", code, str(so)], check=True, stdout=subprocess.PIPE, text=True,
                         env={**os.environ, "LD_PRELOAD": str(so)}, timeout=300).stdout
    made, gone, busy = json.loads(out.strip().splitlines()[-1])
    assert made >= 14 and gone == made and busy == 0, (made, gone, busy)
