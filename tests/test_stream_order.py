"""Every entry point that takes torch tensors waits for the work torch has queued on them (CPU).

A context works on its own stream, which does not wait for torch's.  Stand-ins for the
library and for CUDA tensors record, for each argument that may be a tensor, inputs and
outputs alike, whether torch's current stream of its device was waited for before the
library was called."""
import ctypes as C

import numpy as np
import pytest

NX, NZ, NT, NREC = 20, 16, 12, 5


class _Tensor:
    def __init__(self, n, device="cuda:1"):
        self.n, self.device, self.is_cuda = n, device, True
        self.buf = np.zeros(n, np.float32)

    def is_contiguous(self):
        return True

    def numel(self):
        return self.n

    def data_ptr(self):
        return self.buf.ctypes.data


_Tensor.__module__ = "torch.stand_in"


class _Lib:
    def __init__(self, log):
        self.log = log

    def __getattr__(self, name):
        def call(*a):
            self.log.append(name)
            return 0
        return call


def _calls(ertm):
    """name -> (sizes of the array arguments, call of them)"""
    n, d = NX * NZ, 3 * NT * NREC
    cfg = ertm.Config(nx=NX, ny=1, nz=NZ, dx=10, dy=10, dz=10, dt_ms=1.0, nt=NT, pml=(4, 4, 0, 0, 4, 4))

    def ctx(lib):
        c = object.__new__(ertm.Context)
        c.cfg, c._L, c._h = cfg, lib, C.c_void_p(1)
        c.close = lambda: None
        return c

    def shot(w=None):
        return ertm.Shot(8, 0, 6, wavelet=np.ones(4, np.float32) if w is None else w, rx0=5, nrx=NREC, rz=6)

    win = ertm.Window(0, 0, NX, 1, NT)
    return {
        "set_model": ([n] * 3, lambda L, a: ctx(L).set_model(0, *a)),
        "modelling": ([d, 4], lambda L, a: ctx(L).forward_together_using_real_model(shot(a[1]), out=a[0])),
        "source pass": ([4], lambda L, a: ctx(L).forward_together_using_smoothed_model(shot(a[0]))),
        "receiver pass": ([d, n, n, n], lambda L, a: ctx(L).backward_together_using_smoothed_model(shot(), *a)),
        "rtm_shot": ([d, n, n, n, 4], lambda L, a: ctx(L).rtm_shot(shot(a[4]), *a[:4])),
        "rtm_batch": ([d, d, n, n, n, 4],
                      lambda L, a: ctx(L).rtm_batch([shot(a[5]), shot()], list(a[:2]), *a[2:5])),
        "get_wavefield": ([n], lambda L, a: ctx(L).get_wavefield("vx", out=a[0])),
        "propagate": ([4], lambda L, a: ctx(L).propagate(0, shot(a[0]), 3)),
        "time_kernels": ([4], lambda L, a: ctx(L).time_kernels(shot(a[0]), 3)),
        "born_forward": ([n, n, n, d, 4], lambda L, a: ctx(L).born_forward(shot(a[4]), *a[:4])),
        "born_adjoint": ([d, n, n, n, 4], lambda L, a: ctx(L).born_adjoint(shot(a[4]), *a[:4])),
        "born_forward_shots": ([n, n, n, 2 * d, 4],
                               lambda L, a: ctx(L).born_forward_shots([shot(), shot(a[4])], *a[:4])),
        "born_adjoint_shots": ([2 * d, n, n, n, 4],
                               lambda L, a: ctx(L).born_adjoint_shots([shot(), shot(a[4])], *a[:4])),
        "rtm_multi": ([d, d, n, n, n, 4],
                      lambda L, a: ertm.rtm_multi([ctx(L), ctx(L)], [shot(a[5]), shot()], list(a[:2]),
                                                  [tuple(a[2:5]), tuple(np.zeros(n, np.float32) for _ in range(3))])),
        "rtm_windows": ([n, n, n, d, n, n, n, 4],
                        lambda L, a: ertm.rtm_windows(cfg, *a[:3], [win], [shot(a[7])], [a[3]], 1, *a[4:7])),
        "noalloc": ([n, n, n, d, 4],
                    lambda L, a: ertm.forward_together_using_real_model_noalloc(cfg, *a[:3], shot(a[4]), a[3])),
    }


NAMES = ("set_model", "modelling", "source pass", "receiver pass", "rtm_shot", "rtm_batch", "get_wavefield",
         "propagate", "time_kernels", "born_forward", "born_adjoint", "born_forward_shots", "born_adjoint_shots",
         "rtm_multi", "rtm_windows", "noalloc")


@pytest.mark.parametrize("name", NAMES)
def test_waits_for_every_tensor(ertm, monkeypatch, name):
    import torch
    calls = _calls(ertm)
    assert set(calls) == set(NAMES)
    sizes, call = calls[name]
    for k in range(len(sizes)):
        log = []

        class Stream:
            def __init__(self, device):
                self.device = device

            def synchronize(self):
                log.append(f"wait {self.device}")

        monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: Stream(device))
        lib = _Lib(log)
        monkeypatch.setattr(ertm, "lib", lambda: lib)
        call(lib, [_Tensor(m) if q == k else np.zeros(m, np.float32) for q, m in enumerate(sizes)])
        assert log[0] == "wait cuda:1" and any(e.startswith("ertm_") for e in log[1:]), (name, k, log)
        log.clear()
        call(lib, [np.zeros(m, np.float32) for m in sizes])
        assert not any(e.startswith("wait") for e in log)      # host arrays: nothing to wait for
