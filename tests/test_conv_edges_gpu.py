"""The convolutions, their gradients and the elementwise kernels at the edges of their
tiles, against PyTorch FP32 on the same BF16 inputs (GPU).

Tolerances: a BF16 output is within half a unit in the last place of the FP32 result,
2^-9 relative per element (2^-8 with room for a sum that rounds the other way), so 2^-8 in
relative L2; FP32 weight gradients sum at most 5,000 products of exact BF16 factors here,
each addition within 2^-24: 1e-4.  (PyTorch's TF32 convolutions are exact on BF16 factors.)"""
import ctypes as C
import importlib

import pytest

pytestmark = pytest.mark.gpu

PKG = "2d_and_3d_elastic_reverse_time_migration_b200"
BF16 = 2.0 ** -8


@pytest.fixture(scope="module")
def env():
    import torch
    nn = importlib.import_module(PKG + ".nn")
    dev = torch.device("cuda", 0)
    torch.manual_seed(1)
    return torch, nn, nn.Ops(dev), dev


def _rel(a, b):
    a, b = a.detach().double(), b.detach().double()
    return float((a - b).norm() / b.norm())


def _nchw(t):
    return t.permute(0, 3, 1, 2)


# one pixel; images narrower, one short of, equal to and past the 254-pixel row of a tile;
# channel counts that fill no swizzle span, one, several, and more than one output block
@pytest.mark.parametrize("n,h,w,ci,co", [
    (1, 1, 1, 32, 48), (3, 5, 13, 8, 16), (2, 7, 61, 24, 40), (1, 3, 253, 16, 64), (1, 2, 255, 48, 272),
    (1, 3, 300, 64, 32), (2, 2, 31, 288, 16), (5, 9, 17, 128, 128), (1, 65, 3, 40, 8)])
def test_conv_edges(env, n, h, w, ci, co):
    torch, nn, ops, dev = env
    F = torch.nn.functional
    off, cs = 8, co + 16                       # outputs inside a wider tensor
    x = torch.randn(n, h, w, ci, device=dev).bfloat16()
    wt = (torch.randn(co, 9 * ci, device=dev) * 0.1).bfloat16()
    bias = torch.randn(co, device=dev)
    y = torch.full((n, h, w, cs), 7.0, device=dev, dtype=torch.bfloat16)
    ops.conv(nn.act(x, n, h, w), wt, bias, nn.act(y, n, h, w, co, off), relu=True)
    w4 = wt.float().view(co, 3, 3, ci).permute(0, 3, 1, 2).clone().requires_grad_(True)
    xr = _nchw(x.float()).requires_grad_(True)
    pre = F.conv2d(xr, w4, None, padding=1)
    ref = F.relu(pre.detach() + bias.view(1, -1, 1, 1))
    assert _rel(_nchw(y[..., off:off + co].float()), ref) <= BF16
    assert bool((y[..., :off] == 7).all()) and bool((y[..., off + co:] == 7).all())
    y32 = torch.zeros(n, h, w, co, device=dev)
    ops.conv(nn.act(x, n, h, w), wt, bias, nn.act(y32, n, h, w), relu=False, y32=y32)
    assert _rel(_nchw(y32), pre.detach() + bias.view(1, -1, 1, 1)) <= 1e-5
    dy = torch.zeros(n, h, w, cs, device=dev, dtype=torch.bfloat16)
    dy[..., off:off + co] = torch.randn(n, h, w, co, device=dev)
    dyv = dy[..., off:off + co].float()
    pre.backward(_nchw(dyv))
    wf = torch.zeros(ci, 9 * co, device=dev, dtype=torch.bfloat16)
    ops.flip3(wt, wf, co, ci)
    dx = torch.zeros_like(x)
    ops.conv_dgrad(nn.act(dy, n, h, w, co, off), wf, nn.act(dx, n, h, w), mask=nn.act(x, n, h, w))
    assert _rel(_nchw(dx.float()), xr.grad * (xr.detach() > 0)) <= BF16
    dw = torch.ones(co, 9 * ci, device=dev)    # accumulated
    ops.conv_wgrad(nn.act(x, n, h, w), nn.act(dy, n, h, w, co, off), dw)
    assert _rel(dw.view(co, 3, 3, ci).permute(0, 3, 1, 2) - 1, w4.grad) <= 1e-4
    db = torch.zeros(co, device=dev)
    ops.bias_grad(nn.act(dy, n, h, w, co, off), db)
    assert _rel(db, dyv.sum(dim=(0, 1, 2))) <= 1e-4
    assert int(ops.err.item()) == 0


@pytest.mark.parametrize("n,h,w,ci,co", [(1, 1, 1, 8, 8), (2, 3, 7, 24, 40), (1, 2, 129, 64, 32), (3, 9, 33, 128, 64)])
def test_up2_edges(env, n, h, w, ci, co):
    torch, nn, ops, dev = env
    F = torch.nn.functional
    off, cs = 8, co + 24
    x = torch.randn(n, h, w, ci, device=dev).bfloat16()
    u = (torch.randn(4 * co, ci, device=dev) * 0.1).bfloat16()
    bias = torch.randn(co, device=dev)
    y = torch.full((n, 2 * h, 2 * w, cs), 7.0, device=dev, dtype=torch.bfloat16)
    ops.up(nn.act(x, n, h, w), u, bias, nn.act(y, n, 2 * h, 2 * w, co, off), relu=False)
    wt = u.float().view(2, 2, co, ci).permute(3, 2, 0, 1).contiguous().requires_grad_(True)
    xr = _nchw(x.float()).requires_grad_(True)
    ref = F.conv_transpose2d(xr, wt, None, stride=2)
    assert _rel(_nchw(y[..., off:off + co].float()), ref + bias.view(1, -1, 1, 1)) <= BF16
    assert bool((y[..., :off] == 7).all()) and bool((y[..., off + co:] == 7).all())
    dy = torch.randn(n, 2 * h, 2 * w, cs, device=dev).bfloat16()
    ref.backward(_nchw(dy[..., off:off + co].float()))
    ut = torch.zeros(ci, 4 * co, device=dev, dtype=torch.bfloat16)
    ops.transpose(u, ut, 4 * co, ci)
    dx = torch.zeros_like(x)
    dya = nn.act(dy, n, 2 * h, 2 * w, co, off)
    ops.up_dgrad(dya, ut, nn.act(dx, n, h, w), mask=nn.act(x, n, h, w))
    assert _rel(_nchw(dx.float()), xr.grad * (xr.detach() > 0)) <= BF16
    du = torch.zeros(4 * co, ci, device=dev)
    ops.up_wgrad(nn.act(x, n, h, w), dya, du)
    assert _rel(du.view(2, 2, co, ci).permute(3, 2, 0, 1), wt.grad) <= 1e-4
    assert int(ops.err.item()) == 0


# the vector kernels (16-byte aligned dense operand) against the scalar ones, bit for bit
@pytest.mark.parametrize("n,h,w,c", [(1, 2, 2, 8), (2, 6, 10, 24), (3, 4, 130, 136)])
def test_pool_vector_equals_scalar(env, n, h, w, c):
    torch, nn, ops, dev = env
    x = torch.randn(n, h, w, c + 8, device=dev).bfloat16()
    x[0, 0, :2] = -3.0e38                      # below every other value: the window has no maximum
    xa = nn.act(x, n, h, w, c, 8)
    size = n * (h // 2) * (w // 2) * c
    flat = [torch.zeros(size + 1, device=dev, dtype=torch.bfloat16)[k:k + size] for k in (0, 1)]
    for f in flat:
        ops.pool(xa, f)
    assert torch.equal(*flat)
    dy = torch.randn(size, device=dev).bfloat16()
    off = torch.zeros(size + 1, device=dev, dtype=torch.bfloat16)[1:]
    off.copy_(dy)
    for mask in (False, True):
        dx = [torch.ones_like(x) for _ in range(2)]
        for d, g in zip(dx, (dy, off)):
            ops.pool_bwd(xa, g, nn.act(d, n, h, w, c, 8), relu_mask=mask)
        assert torch.equal(*dx)


# one packed pass from a dense FP32 input against the general path (views, other types)
@pytest.mark.parametrize("n,h,w", [(1, 8, 8), (2, 16, 24)])
def test_op_lists(env, n, h, w):
    torch, nn, ops, dev = env
    net = nn.UNet(dev, seed=2)
    x = torch.randn(n, h, w, 3, device=dev)
    want = net.forward(x).clone()
    wide = torch.randn(n, h, w, 5, device=dev)
    wide[..., 1:4] = x
    for other in (wide[..., 1:4], x.double(), x.cpu()):
        assert torch.equal(net.forward(other), want)
    B, G = net._buffers(n, h, w)
    o, P = net.ops, net.params                 # the first layers one by one
    ea, eb = torch.zeros_like(B["e0a"]), torch.zeros_like(B["cat0"])
    o.conv(nn.act(B["in0"], n, h, w), P["e0a"].wb, P["e0a"].b, nn.act(ea, n, h, w))
    o.conv(nn.act(ea, n, h, w), P["e0b"].wb, P["e0b"].b, nn.act(eb, n, h, w, 16, 16))
    assert torch.equal(ea, B["e0a"]) and torch.equal(eb[..., 16:], B["cat0"][..., 16:])
    g = torch.randn(n, h, w, nn.OUT_P, device=dev).bfloat16()
    for p in P.values():
        p.g.fill_(3.0)                         # zeroed by the pass
        p.bg.fill_(3.0)
    net.backward(g)
    dw, db = torch.zeros_like(P["out"].g), torch.zeros_like(P["out"].bg)
    o.conv_wgrad(nn.act(B["d0b"], n, h, w), nn.act(g, n, h, w), dw)
    o.bias_grad(nn.act(g, n, h, w), db)
    assert _rel(P["out"].g, dw) <= 1e-5 and _rel(P["out"].bg, db) <= 1e-5
    # refused: an unknown operation, a pointer outside the table
    L = nn.lib()
    ptr, done = (C.c_void_p * 1)(x.data_ptr()), C.c_int(9)
    op = type(net._buffers(n, h, w).fwd.ops[0])()
    for kind, p0 in ((99, 0), (nn.ZERO, 1), (nn.ZERO, -1)):
        op.kind, op.n = kind, 4
        op.p[0] = p0
        rc = L.ertm_nn_run(C.byref(op), 1, ptr, 1, C.byref(done), None, o.st)
        assert rc == -1 and done.value == 0
    assert int(o.err.item()) == 0


# splitk bounds the partial sums of an element; one sum is repeatable, with any number of pixels
@pytest.mark.parametrize("n,h,w,ci,co", [(2, 7, 61, 24, 40), (3, 40, 130, 32, 48), (2, 64, 128, 16, 16),
                                         (1, 33, 70, 128, 64)])
def test_one_sum_per_weight_is_repeatable(env, n, h, w, ci, co):
    torch, nn, ops, dev = env
    x = torch.randn(n, h, w, ci, device=dev).relu().bfloat16()
    dy, dyu = (torch.randn(n, s * h, s * w, co, device=dev).bfloat16() for s in (1, 2))

    def grads(k):
        dw, du = torch.zeros(co, 9 * ci, device=dev), torch.zeros(4 * co, ci, device=dev)
        ops.conv_wgrad(nn.act(x, n, h, w), nn.act(dy, n, h, w), dw, splitk=k)
        ops.up_wgrad(nn.act(x, n, h, w), nn.act(dyu, n, 2 * h, 2 * w), du, splitk=k)
        return dw, du

    first, many = grads(1), grads(0)
    for _ in range(20):
        assert all(torch.equal(a, b) for a, b in zip(grads(1), first))
    for k in (2, 5):                           # as the other splits, to the FP32 rounding of the sums
        for a, b in zip(grads(k), many):
            assert _rel(a, b) <= 1e-4
    for a, b in zip(first, many):
        assert _rel(a, b) <= 1e-4
    assert int(ops.err.item()) == 0


def _conv64(torch, x, wt, taps):
    """y (n, h, w, co) of x (n, h, w, ci) and weights (co, taps, ci) in 64 bits on the CPU, one output
    pixel's own taps only (zero padding)."""
    F = torch.nn.functional
    n, h, w, ci = x.shape
    cols = F.unfold(_nchw(x.double().cpu()), 3, padding=1).view(n, ci, taps, h * w).permute(0, 3, 2, 1)
    return (cols.reshape(n * h * w, -1) @ wt.double().cpu().view(wt.shape[0], -1).T).view(n, h, w, -1)


def _same_kind(torch, got, ref, tol):
    """NaN and infinities at the same places, the finite rest within tol in relative L2"""
    got, ref = got.double().cpu(), ref.double().cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(ref))
    inf = torch.isinf(ref)
    assert torch.equal(torch.isinf(got), inf) and torch.equal(got[inf], ref[inf])
    f = torch.isfinite(ref)
    assert bool(f.any()) and float((got[f] - ref[f]).norm()) <= tol * float(ref[f].norm())


# an infinite or NaN input reaches the outputs that have it under one of their taps, and no
# other; channel counts of every way to stage them (one chunk, swizzled, chunk planes, streamed)
@pytest.mark.parametrize("n,h,w,ci,co", [(1, 9, 13, 8, 16), (2, 12, 128, 8, 16), (1, 6, 300, 8, 24), (1, 9, 13, 24, 16),
                                         (1, 7, 128, 16, 16), (1, 11, 40, 48, 32), (1, 6, 21, 288, 16)])
def test_conv_keeps_nonfinite_inputs_local(env, n, h, w, ci, co):
    torch, nn, ops, dev = env
    x = torch.randn(n, h, w, ci, device=dev).bfloat16()
    x[0, h - 1, w - 1, 3], x[0, 4, 7, 0], x[0, 0, 0, 5] = float("inf"), float("nan"), float("-inf")
    wt = (0.5 + torch.rand(co, 9 * ci, device=dev)).bfloat16()
    y = torch.zeros(n, h, w, co, device=dev)
    ops.conv(nn.act(x, n, h, w), wt, None, nn.act(y, n, h, w), relu=False, y32=y)
    _same_kind(torch, y, _conv64(torch, x, wt, 9), 1e-5)
    assert int(ops.err.item()) == 0


# the same of the weight gradients, with infinite and NaN activations in the last row and column,
# where a tile's dy ends in zeros, and infinite gradients beside the padding
@pytest.mark.parametrize("n,h,w,ci,co", [(1, 1, 1, 8, 8), (1, 9, 13, 8, 16), (2, 12, 128, 16, 16), (1, 7, 40, 64, 32),
                                         (1, 5, 300, 24, 40), (3, 33, 64, 32, 48), (2, 6, 31, 128, 144)])
@pytest.mark.parametrize("splitk", [0, 1])
def test_wgrad_keeps_nonfinite_inputs_local(env, n, h, w, ci, co, splitk):
    torch, nn, ops, dev = env
    x = torch.randn(n, h, w, ci, device=dev).bfloat16()
    dy = (0.5 + torch.rand(n, h, w, co, device=dev)).bfloat16()
    x[n - 1, h - 1, w - 1, 0], x[0, h // 2, w - 1, 1] = float("inf"), float("-inf")
    x[0, h - 1, w // 2, 2], x[0, 0, 0, 3] = float("nan"), float("inf")
    dy[0, 0, w // 2, 4], dy[n - 1, h - 1, w - 1, 5] = float("inf"), float("nan")
    dw = torch.zeros(co, 9 * ci, device=dev)
    ops.conv_wgrad(nn.act(x, n, h, w), nn.act(dy, n, h, w), dw, splitk=splitk)
    cols = torch.nn.functional.unfold(_nchw(x.double().cpu()), 3, padding=1).view(n, ci, 9, h * w)
    ref = torch.einsum("nctp,npo->otc", cols, dy.double().cpu().view(n, h * w, co))
    _same_kind(torch, dw.view(co, 9, ci), ref, 1e-4)
    dyu = (0.5 + torch.rand(n, 2 * h, 2 * w, co, device=dev)).bfloat16()
    dyu[0, 1, 2 * w - 1, 4], dyu[n - 1, 2 * h - 1, 0, 5] = float("inf"), float("nan")
    du = torch.zeros(4 * co, ci, device=dev)
    ops.up_wgrad(nn.act(x, n, h, w), nn.act(dyu, n, 2 * h, 2 * w), du, splitk=splitk)
    g = dyu.double().cpu().view(n, h, 2, w, 2, co).permute(0, 1, 3, 2, 4, 5).reshape(n * h * w, 4 * co)
    _same_kind(torch, du, g.T @ x.double().cpu().view(n * h * w, ci), 1e-4)
    assert int(ops.err.item()) == 0
