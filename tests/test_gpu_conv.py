"""The implicit-GEMM convolution kernels (maf_nn_conv, maf_nn_conv_wgrad) against FP64
convolutions of the same BF16 values: tiles that end inside an image row, rows shorter
than a copy step, channel counts that leave part of a K block or of an output tile
empty, more tiles than resident CTAs, every output tile width.  FP32 accumulation in steps
of 16 exact products, each step at most one unit in the last place (2^-23) of the running
sum: up to 108 steps (K <= 1728) forward, and for the weights 64 steps of a slab plus the
64 slabs, i.e. 1.5e-5 of the sums' size; 3e-5 of the result's largest value."""
import ctypes as C

import pytest

M = pytest.importorskip("magnumaf")
torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

TOL = 3e-5


def _p(t):
    return C.c_void_p(t.data_ptr())


def _act(g, B, H, W, c, cp):
    a = torch.zeros(B, H, W, cp, device="cuda", dtype=torch.bfloat16)
    a[..., :c] = torch.randn(B, H, W, c, device="cuda", generator=g).to(torch.bfloat16)
    return a


@pytest.mark.parametrize("B,H,W,cin,cout", [(1, 16, 16, 8, 32), (1, 4, 4, 24, 16), (3, 12, 20, 5, 3), (2, 16, 24, 96, 64),
                                            (1, 8, 8, 192, 128), (1, 32, 32, 64, 192), (4, 128, 128, 32, 32)])
def test_conv_and_weight_gradient(B, H, W, cin, cout):
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + H * 10 + cin)
    cp, coutp, P = -(-cin // 8) * 8, -(-cout // 8) * 8, B * H * W
    act = _act(g, B, H, W, cin, cp)
    w32 = torch.randn(cout, 9, cin, device="cuda", generator=g)
    wf = torch.empty(cout, 9 * cp, device="cuda", dtype=torch.bfloat16)
    wd = torch.empty(cin, 9 * coutp, device="cuda", dtype=torch.bfloat16)
    M._ck(M.lib.maf_nn_wcast_conv(_p(w32), cout, cin, cp, coutp, _p(wf), _p(wd), None))
    bias = torch.randn(cout, device="cuda", generator=g)
    out = torch.full((P, cout), float("nan"), device="cuda")
    outb = torch.full((P, coutp), float("nan"), device="cuda", dtype=torch.bfloat16)
    M._ck(M.lib.maf_nn_conv(_p(act), B, H, W, cp, _p(wf), cout, _p(bias), 1, _p(out), cout, _p(outb), coutp, None))
    torch.cuda.synchronize()
    x = act[..., :cin].double().permute(0, 3, 1, 2)
    w = w32.to(torch.bfloat16).double().reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
    ref = torch.nn.functional.conv2d(x, w, bias.double(), padding=1).relu().permute(0, 2, 3, 1).reshape(P, cout)
    assert (out.double() - ref).abs().max() <= TOL * ref.abs().max()
    assert torch.equal(outb[:, :cout], out.to(torch.bfloat16)) and not outb[:, cout:].any()
    # data gradient: the same kernel on dY with the flipped weights
    dy = torch.zeros(B, H, W, coutp, device="cuda", dtype=torch.bfloat16)
    dy[..., :cout] = torch.randn(B, H, W, cout, device="cuda", generator=g).to(torch.bfloat16)
    dx = torch.full((P, cin), float("nan"), device="cuda")
    M._ck(M.lib.maf_nn_conv(_p(dy), B, H, W, coutp, _p(wd), cin, None, 0, _p(dx), cin, None, 0, None))
    # weight gradient
    work = torch.empty(64 * 9 * cp * coutp, device="cuda")
    dw = torch.full((cout, 9, cin), float("nan"), device="cuda")
    M._ck(M.lib.maf_nn_conv_wgrad(_p(act), B, H, W, cp, cin, _p(dy), cout, coutp, _p(work), 64, _p(dw), None))
    torch.cuda.synchronize()
    d = dy[..., :cout].double().permute(0, 3, 1, 2)
    rx = torch.nn.grad.conv2d_input(x.shape, w, d, padding=1).permute(0, 2, 3, 1).reshape(P, cin)
    rw = torch.nn.grad.conv2d_weight(x, w.shape, d, padding=1).permute(0, 2, 3, 1).reshape(cout, 9, cin)
    assert (dx.double() - rx).abs().max() <= TOL * rx.abs().max()
    assert (dw.double() - rw).abs().max() <= TOL * rw.abs().max()


def test_conv_rejects_bad_arguments():
    a = torch.zeros(64, 8, device="cuda", dtype=torch.bfloat16)
    o = torch.zeros(64, 32, device="cuda")
    assert M.lib.maf_nn_conv(_p(a), 1, 8, 8, 12, _p(a), 8, None, 0, _p(o), 8, None, 0, None) == 1  # Cp not a multiple of 8
    assert M.lib.maf_nn_conv(_p(a), 1, 8, 8, 8, _p(a), 8, None, 0, _p(o), 4, None, 0, None) == 1   # ldo below N
    assert M.lib.maf_nn_conv(C.c_void_p(a.data_ptr() + 2), 1, 8, 8, 8, _p(a), 8, None, 0, _p(o), 8, None, 0, None) == 1


@pytest.mark.parametrize("P,c", [(1, 3), (100, 8), (5000, 24), (4096, 264)])
def test_relu_and_bias_gradient(P, c):
    g = torch.Generator(device="cuda").manual_seed(P + c)
    cp = -(-c // 8) * 8
    dA = torch.randn(P, c, device="cuda", generator=g)
    A = torch.randn(P, c, device="cuda", generator=g).relu()
    n = C.c_int()
    M._ck(M.lib.maf_nn_relu_bias_bwd_parts(C.byref(n)))
    part = torch.empty(n.value * c, device="cuda", dtype=torch.float64)
    dyb = torch.full((P, cp), float("nan"), device="cuda", dtype=torch.bfloat16)
    db = torch.empty(c, device="cuda")
    M._ck(M.lib.maf_nn_relu_bias_bwd(_p(dA), _p(A), P, c, 1, _p(dyb), cp, _p(db), _p(part), None))
    torch.cuda.synchronize()
    ref = dA * (A > 0)
    assert torch.equal(dyb[:, :c], ref.to(torch.bfloat16)) and not dyb[:, c:].any()
    # FP64 sums of FP32 values, rounded once
    s = ref.double().sum(0)
    assert ((db.double() - s).abs() <= 1.2e-7 * s.abs() + 1e-12 * ref.abs().double().sum(0)).all()
