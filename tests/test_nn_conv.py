"""The convolution kernels over the edges of their tiles: partial 8 x 16 tiles,
grids below a tile, every padding, input channels beyond the view, output
channels that are no multiple of 8 or 16 and more than one slice, narrow and
wide inputs.  The reference is the same sum in FP64 on the BF16 operands."""
import ctypes as C

import numpy as np
import pytest

# nx, ny, nz, xper, yper, channels of the input (split: a second view from channel
# c1 on), Kc, co, Np, relu, mask
CASES = [
    (8, 16, 4, 1, 1, 16, 16, 16, 16, 1, 0),       # one tile
    (4, 4, 2, 1, 1, 8, 16, 3, 16, 0, 0),          # below a tile, head
    (5, 3, 1, 0, 1, 24, 32, 24, 32, 1, 1),        # one plane, ragged
    (9, 17, 7, 1, 0, 24, 32, 20, 32, 0, 0),       # one point over a tile
    (23, 37, 11, 0, 0, 72, 80, 24, 32, 1, 0),     # wide input, bounded
    (16, 33, 5, 1, 1, 48, 48, 192, 192, 1, 1),    # several slices
    (24, 16, 19, 1, 1, 32, 32, 72, 80, 0, 1),     # 80 columns
    (10, 18, 6, 1, 1, 96, 96, 96, 96, 1, 0),
    (17, 9, 5, 0, 1, 192, 192, 192, 192, 1, 1),   # wide on both sides
    (9, 20, 6, 1, 0, 240, 240, 48, 48, 0, 0),
    (8, 8, 4, 1, 1, 104, 112, 45, 48, 1, 0),
    (12, 6, 3, 1, 1, 200, 256, 256, 256, 1, 0),   # the largest channel counts
    (64, 48, 40, 1, 1, 24, 32, 24, 32, 1, 1),     # several items a CTA
    (20, 17, 5, 1, 0, (48, 24), 80, 24, 32, 1, 0),     # two views, resident weights
    (9, 8, 6, 1, 1, (24, 60), 96, 20, 32, 0, 1),
    (16, 18, 4, 0, 1, (192, 48), 240, 48, 48, 1, 0),   # two views, streamed weights
]


def _reference(x, W, b, xper, yper):
    """sum over taps in FP64; x [nx, ny, nz, c], W [27, co, c]"""
    nx, ny, nz, c = x.shape
    xp = np.zeros((nx + 2, ny + 2, nz + 2, c))
    xp[1:-1, 1:-1, 1:-1] = x
    if xper:
        xp[0], xp[-1] = xp[-2], xp[1]
    if yper:
        xp[:, 0], xp[:, -1] = xp[:, -2], xp[:, 1]
    y = np.zeros((nx, ny, nz, W.shape[1]))
    s = np.zeros_like(y)
    for t in range(27):
        dk, dj, di = t // 9, t // 3 % 3, t % 3
        v = xp[di:di + nx, dj:dj + ny, dk:dk + nz]
        y += v @ W[t].T
        s += np.abs(v) @ np.abs(W[t]).T
    return y + b, s + np.abs(b)


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_conv(case):
    import torch
    from glemur_gb300 import _abi
    nx, ny, nz, xper, yper, chans, Kc, co, Np, relu, mask = case
    n1, n2 = chans if isinstance(chans, tuple) else (chans, 0)
    c1 = n1 + n2
    rng = np.random.default_rng(1)
    bf = lambda a: torch.tensor(a, dtype=torch.float32, device="cuda").to(torch.bfloat16)  # noqa: E731
    V = nx * ny * nz
    x = bf(rng.normal(size=(V, c1)))
    W = bf(np.pad(rng.normal(size=(27, co, c1)) / np.sqrt(27 * c1), ((0, 0), (0, Np - co), (0, Kc - c1))))
    b = torch.tensor(np.pad(rng.normal(size=co), (0, Np - co)), dtype=torch.float32, device="cuda")
    lo = (co + 7) // 8 * 8 + 8
    y = torch.full((V, lo), 7.0, dtype=torch.bfloat16, device="cuda")
    m = bf(rng.normal(size=(V, lo)))
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    l2 = (n2 + 7) // 8 * 8 + 8
    x1, x2 = x[:, :n1].contiguous(), torch.nn.functional.pad(x[:, n1:], (0, l2 - n2), value=9.0)
    torch.cuda.synchronize()
    lib = _abi.load()
    _abi.check(lib.gm_nn_conv(P(x1), n1, n1, P(x2) if n2 else None, l2, n2, P(W), C.cast(b.data_ptr(), C.POINTER(C.c_float)), P(y), lo, co,
                              P(m) if mask else None, lo if mask else 0, relu, nx, ny, nz, xper, yper, Kc, Np, P(st),
                              None), "gm_nn_conv")
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    xs = x.double().cpu().numpy().reshape(nz, ny, nx, c1).transpose(2, 1, 0, 3)
    ref, size = _reference(xs, W.double().cpu().numpy()[:, :co, :c1], b.double().cpu().numpy()[:co], xper, yper)
    if relu:
        ref = np.maximum(ref, 0)
    if mask:
        ms = m.double().cpu().numpy()[:, :co].reshape(nz, ny, nx, co).transpose(2, 1, 0, 3)
        ref = np.where(ms > 0, ref, 0)
    got = y.double().cpu().numpy()
    g = got[:, :co].reshape(nz, ny, nx, co).transpose(2, 1, 0, 3)
    # FP32 sums of 27 Kc products (each addition off by at most an ulp of the sum
    # of magnitudes) and one rounding to BF16 (2^-9 relative)
    tol = size * (27 * Kc * 2.0 ** -23) + np.abs(ref) * 2.0 ** -8
    assert np.all(np.abs(g - ref) <= tol), np.max(np.abs(g - ref) / tol)
    assert np.all(got[:, co:] == 7.0)          # nothing beyond the output's channels


# nx, ny, nz, xper, yper, ci, co, chunk: ragged tiles, blocks of fewer planes at the
# end, several slices of input and output channels, several blocks a CTA
WGRAD_CASES = [
    (17, 33, 9, 1, 1, 20, 20, 0),
    (9, 16, 5, 0, 1, 44, 100, 0),
    (24, 31, 7, 1, 0, 96, 49, 4096),
    (32, 32, 33, 1, 1, 3, 24, 16384),
    (7, 5, 1, 0, 0, 120, 16, 0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", WGRAD_CASES, ids=lambda c: "x".join(map(str, c)))
def test_conv_wgrad(case):
    import torch
    from glemur_gb300 import _abi
    nx, ny, nz, xper, yper, ci, co, chunk = case
    rng = np.random.default_rng(2)
    V, ldi, ldo = nx * ny * nz, (ci + 7) // 8 * 8 + 8, (co + 7) // 8 * 8
    bf = lambda a: torch.tensor(a, dtype=torch.float32, device="cuda").to(torch.bfloat16)  # noqa: E731
    x, d = bf(rng.normal(size=(V, ldi))), bf(rng.normal(size=(V, ldo)))
    dW = torch.zeros(27, co, ci, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    torch.cuda.synchronize()
    lib = _abi.load()
    _abi.check(lib.gm_nn_conv_wgrad(P(d), ldo, co, P(x), ldi, ldi, None, 0, 0, C.cast(dW.data_ptr(), C.POINTER(C.c_float)),
                                    ci, nx, ny, nz, xper, yper, chunk, P(st), None), "gm_nn_conv_wgrad")
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    xs = x.double().cpu().numpy()[:, :ci].reshape(nz, ny, nx, ci).transpose(2, 1, 0, 3)
    ds = d.double().cpu().numpy()[:, :co].reshape(nz, ny, nx, co).transpose(2, 1, 0, 3).reshape(V, co)
    xp = np.zeros((nx + 2, ny + 2, nz + 2, ci))
    xp[1:-1, 1:-1, 1:-1] = xs
    if xper:
        xp[0], xp[-1] = xp[-2], xp[1]
    if yper:
        xp[:, 0], xp[:, -1] = xp[:, -2], xp[:, 1]
    got = dW.double().cpu().numpy()
    for t in range(27):
        dk, dj, di = t // 9, t // 3 % 3, t % 3
        v = xp[di:di + nx, dj:dj + ny, dk:dk + nz].reshape(V, ci)
        ref, size = ds.T @ v, np.abs(ds).T @ np.abs(v)
        # an FP32 sum of V exact products: each addition off by at most an ulp of the sum of magnitudes
        assert np.all(np.abs(got[t] - ref) <= size * V * 2.0 ** -23), t


# channels, channel stride: 16-byte rows of whole groups of 8, and what falls short of that
PASSES = [(24, 24), (48, 72), (3, 8), (20, 24), (8, 9), (264, 264), (1030, 1030)]


@pytest.mark.gpu
@pytest.mark.parametrize("c,ld", PASSES)
def test_elementwise_passes(c, ld):
    """Pooling, upsampling, ReLU and bias gradients: one rounding to BF16 of FP32 sums of at most 9
    terms, and an FP32 sum over the voxels."""
    import torch
    from glemur_gb300 import _abi
    lib = _abi.load()
    nx, ny, nz = 6, 10, 4
    V, Vc = nx * ny * nz, nx * ny * nz // 8
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda n: torch.randn(n, ld, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    fine, coarse, y = r(V), r(Vc), r(V)

    def blocks(t):           # [Vc, 8, ld]
        return t.view(nz // 2, 2, ny // 2, 2, nx // 2, 2, ld).permute(0, 2, 4, 1, 3, 5, 6).reshape(Vc, 8, ld)

    def same(got, want, before):
        tol = want.abs() * 2.0 ** -8 + 1e-6
        assert bool(((got[..., :c].double() - want[..., :c]).abs() <= tol[..., :c]).all())
        assert torch.equal(got[..., c:], before[..., c:])

    def run(name, *a):
        _abi.check(getattr(lib, name)(*a, None), name)
        torch.cuda.synchronize()

    torch.cuda.synchronize()
    o = coarse.clone()
    run("gm_nn_pool", P(fine), ld, P(o), ld, c, nx, ny, nz, 0, 0)
    same(o, blocks(fine).double().mean(1), coarse)
    for acc in (0, 1):
        o = fine.clone()
        run("gm_nn_pool", P(coarse), ld, P(o), ld, c, nx, ny, nz, 1, acc)
        same(blocks(o), acc * blocks(fine).double() + coarse.double()[:, None] / 8, blocks(fine))
    o = fine.clone()
    run("gm_nn_upsample", P(coarse), ld, P(o), ld, c, nx, ny, nz, 0)
    same(blocks(o), coarse.double()[:, None].expand(-1, 8, -1), blocks(fine))
    o = coarse.clone()
    run("gm_nn_upsample", P(fine), ld, P(o), ld, c, nx, ny, nz, 1)
    same(o, blocks(fine).double().sum(1), coarse)
    o = fine.clone()
    run("gm_nn_relu_bwd", P(o), ld, P(y), ld, c, V)
    same(o, torch.where(y > 0, fine, torch.zeros_like(fine)).double(), fine)
    db = torch.ones(c + 1, device="cuda")
    run("gm_nn_bias_grad", P(fine), ld, c, V, C.cast(db.data_ptr(), C.POINTER(C.c_float)))
    size = fine.double().abs().sum(0)[:c] + 1
    assert bool(((db[:c].double() - 1 - fine.double().sum(0)[:c]).abs() <= size * V * 2.0 ** -23).all()) and float(db[c]) == 1


def _wgrad(x, d, n, ci, co, xper, yper, chunk):
    """The kernel's gradient of [V, >= ci] inputs and [V, >= co] upstream gradients, and the
    same sums in FP64 by torch."""
    import torch
    from glemur_gb300 import _abi
    nx, ny, nz = n
    dW = torch.zeros(27, co, ci, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    torch.cuda.synchronize()
    _abi.check(_abi.load().gm_nn_conv_wgrad(P(d), d.shape[1], co, P(x), x.shape[1], x.shape[1], None, 0, 0,
                                            C.cast(dW.data_ptr(), C.POINTER(C.c_float)), ci, nx, ny, nz, xper, yper, chunk,
                                            P(st), None), "gm_nn_conv_wgrad")
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    v = torch.zeros(nz + 2, ny + 2, nx + 2, ci, device="cuda", dtype=torch.float64)
    v[1:-1, 1:-1, 1:-1] = x[:, :ci].double().view(nz, ny, nx, ci)
    if xper:
        v[:, :, 0], v[:, :, -1] = v[:, :, -2].clone(), v[:, :, 1].clone()
    if yper:
        v[:, 0], v[:, -1] = v[:, -2].clone(), v[:, 1].clone()
    g = d[:, :co].double()
    ref = torch.stack([g.T @ v[t // 9:t // 9 + nz, t // 3 % 3:t // 3 % 3 + ny, t % 3:t % 3 + nx].reshape(-1, ci) for t in range(27)])
    return dW.double(), ref


@pytest.mark.gpu
@pytest.mark.parametrize("n,ci,co,xper,yper,chunk", [((64, 64, 128), 72, 24, 1, 1, 0), ((64, 64, 128), 3, 24, 1, 1, 0),
                                                     ((60, 50, 75), 24, 20, 0, 1, 65536), ((32, 32, 64), 100, 70, 1, 0, 0),
                                                     ((70, 41, 90), 16, 3, 1, 1, 131072), ((80, 80, 280), 20, 8, 1, 1, 896000)])
def test_conv_wgrad_of_whole_numbers_is_exact(n, ci, co, xper, yper, chunk):
    """Operands -3 .. 3: every partial sum is a whole number below 2^24 (9 x 1,792,000), so a
    lost or doubled tile, plane or chain shows as itself.  Several blocks a chain and
    several chains a block of threads."""
    import torch
    V = n[0] * n[1] * n[2]
    g = torch.Generator(device="cuda").manual_seed(4)
    whole = lambda c: torch.randint(-3, 4, (V, (c + 7) // 8 * 8), device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    got, ref = _wgrad(whole(ci), whole(co), n, ci, co, xper, yper, chunk)
    assert torch.equal(got, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("n,ci,co", [((64, 64, 128), 72, 24), ((128, 128, 256), 72, 24)])
def test_conv_wgrad_error_is_bounded_on_any_grid(n, ci, co):
    """Sums of one sign mostly.  A chain of at most 22,528 voxels is 1408 truncated additions;
    each takes half of 2^-23 of the sum on average, which is half its final value on
    average: 1408 x 2^-23 / 4 = 4.2e-5 of the gradient."""
    import torch
    V = n[0] * n[1] * n[2]
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(V, (ci + 7) // 8 * 8, device="cuda", generator=g).relu().to(torch.bfloat16)
    d = (torch.randn(V, (co + 7) // 8 * 8, device="cuda", generator=g) + 0.3).to(torch.bfloat16)
    got, ref = _wgrad(x, d, n, ci, co, 1, 1, 0)
    assert float((got - ref).norm() / ref.norm()) < 1408 * 2.0 ** -23 / 4
