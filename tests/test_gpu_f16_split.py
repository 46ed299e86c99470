"""Large products (the fp16-split kernels of csrc/matmul_tc_f16.cuh): edges of their tiles, slices and rings, the choice of a row's
scale, and the forms they share with each other."""
import math
import os

import pytest
import torch

from oracle import bounds_oracle as O

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _bound(rows, Di, Do, seed, gap=0.5):
    g = torch.Generator(device=DEV).manual_seed(seed)
    lw = torch.randn(rows, Di, Do, generator=g, device=DEV)
    uw = lw + torch.rand(rows, Di, Do, generator=g, device=DEV) * gap
    lb = torch.randn(rows, Do, generator=g, device=DEV)
    return [lw, uw, lb, lb + torch.rand(rows, Do, generator=g, device=DEV) * gap]


def _weight(N, K, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(N, K, generator=g, device=DEV) / math.sqrt(K), torch.randn(N, generator=g, device=DEV)


def _check(y, lo, up, W, bias, what):
    """Against fp64, entry by entry, within what the arithmetic allows: every product loses at most 2^-21 of itself (two rounded fp16
    parts a side, no product of the small ones) or 2^-27 of the row's largest value (a part at the end of fp16's range, K > 128
    leaving eleven binades above the first 128 values of a row); each of the 3 K / 16 additions to an accumulator truncates at
    2^-23 of it; one rounding at the end."""
    K = W.shape[1]
    c, r = (lo.double() + up.double()) / 2, (up.double() - lo.double()) / 2
    Wd = W.double()
    yc, yr = c @ Wd.t(), r @ Wd.abs().t()
    S = c.abs() @ Wd.abs().t() + r.abs() @ Wd.abs().t()
    top = torch.maximum(lo.abs(), up.abs()).double().amax(-1, keepdim=True)
    bar = S * (2.0 ** -21 + 3 * K / 16 * 2.0 ** -23) + top * (2.0 ** -27 * Wd.abs().sum(1) + 2.0 ** -38 * K * Wd.abs().amax(1)) + 1e-30
    b = 0.0 if bias is None else bias.double()
    for got, ref in ((y[0], yc - yr + b), (y[1], yc + yr + b)):
        d = (got.double() - ref).abs() - bar - 2.0 ** -23 * ref.abs()
        assert bool(torch.isfinite(got).all()), what
        assert float(d.max()) <= 0, (what, float(d.max()))


# rows of weights: at least 296 row tiles of 128 per 128 columns (K <= 128), or 460 800 / K (K >= 320)
@pytest.mark.parametrize("rows,Di,K,N", [(300, 128, 8, 128), (301, 127, 32, 96), (300, 128, 36, 68), (600, 64, 64, 128), (299, 128, 68, 100),
                                         (300, 128, 100, 128), (160, 128, 128, 132), (101, 129, 124, 384), (300, 128, 128, 512),
                                         (480, 128, 320, 260), (1441, 128, 324, 72), (401, 96, 512, 512), (300, 129, 544, 384)])
def test_edges_of_tiles_and_slices(rows, Di, K, N):
    from faith_b200 import _lib, ops
    lw, uw, lb, ub = _bound(rows, Di, K, 5)
    W, bias = _weight(N, K, 6)
    y = ops.matmul(lw, uw, lb, ub, W, bias)
    _check(y[:2], lw, uw, W, None, "weights")
    if rows >= 256:   # (fewer bias rows go to another kernel)
        _check(y[2:], lb, ub, W, bias, "bias terms")
    for _ in range(3):
        for a, b in zip(ops.matmul(lw, uw, lb, ub, W, bias), y):
            assert torch.equal(a, b)
    assert _lib.load().fb_tc_check() == 0


@pytest.mark.parametrize("K,N", [(128, 128), (512, 160)])
def test_rows_and_columns_of_any_magnitude(K, N):
    """Rows of x between 1e-30 and 1e30, rows of W likewise, rows whose values grow by 2^30 along K, that begin with zeros, that are
    zero; the scales are powers of two per row, so only what lies 2^27 below a row's largest value may be lost."""
    from faith_b200 import _lib, ops
    rows, Di = 400 if K == 512 else 300, 256
    lw, uw, lb, ub = _bound(rows, Di, K, 7)
    W, _ = _weight(N, K, 8)
    lw, uw = lw.clone(), uw.clone()
    scale = torch.ones(rows, Di, 1, device=DEV)
    scale[1], scale[2], scale[3] = 1e30, 1e-30, 2.0 ** -100
    grow = torch.ones(rows, Di, K, device=DEV)
    grow[5] = torch.exp2(torch.linspace(-15, 15, K, device=DEV))
    grow[6, ::3, :K // 2] = 0.0
    grow[7] = 0.0
    grow[8, 1::2, 129:] = 2.0 ** 20
    lw, uw = lw * scale * grow, uw * scale * grow
    W = W * torch.exp2(torch.linspace(-20, 20, N, device=DEV)).unsqueeze(1)
    y = ops.matmul(lw, uw, lb, ub, W, None)
    _check(y[:2], lw, uw, W, None, "weights")
    assert bool((y[0][7] == 0).all()) and bool((y[1][7] == 0).all())
    # a value that is not finite spoils its own row and no other
    lw2 = lw.clone()
    lw2[11, 5, 3], lw2[12, 6, K - 1] = float("nan"), float("inf")
    z = ops.matmul(lw2, uw, lb, ub, W, None)
    assert not bool(torch.isfinite(z[0][11, 5]).any()) and not bool(torch.isfinite(z[1][12, 6]).any())
    keep = torch.ones(rows, Di, dtype=torch.bool, device=DEV)
    keep[11, 5] = keep[12, 6] = False
    assert torch.equal(z[0][keep], y[0][keep]) and torch.equal(z[1][keep], y[1][keep])
    assert _lib.load().fb_tc_check() == 0


@pytest.mark.parametrize("S,K,N", [(10, 128, 128), (10, 96, 192), (32, 512, 128)])
def test_forms_agree_bit_for_bit(S, K, N, monkeypatch):
    """Slopes applied while reading, a residual added, bias rows in a launch of their own, one tensor as both lines, ranges returned:
    the same bits as the separate operators at the sizes that take these kernels."""
    from faith_b200 import _lib, ops
    L, Di, p, eps = 32, 128, float("inf"), 0.05
    lw, uw, lb, ub = [t.view(S, L, *t.shape[1:]) for t in _bound(S * L, Di, K, 9)]
    W, bias = _weight(N, K, 10)
    res = [t.view(S, L, *t.shape[1:]) for t in _bound(S * L, Di, N, 11)]
    r = ops.relax(_lib.FB_RELU, lw, uw, lb, ub, p, eps, 1)
    c_l, c_u, nlb, nub = ops.relax_coef(_lib.FB_RELU, lw, uw, lb, ub, p, eps, 1)
    plain = ops.matmul(r[0], r[1], r[2], r[3], W, bias)
    for a, b in zip(ops.matmul_coef(lw, uw, nlb, nub, c_l, c_u, W, bias), plain):
        assert torch.equal(a, b)
    summed = ops.add(plain, res)
    for a, b in zip(ops.matmul_residual(lw, uw, nlb, nub, W, bias, res, c_l, c_u), summed):
        assert torch.equal(a, b)
    for a, b in zip(ops.matmul_residual(r[0], r[1], r[2], r[3], W, bias, res), summed):
        assert torch.equal(a, b)
    monkeypatch.setenv("FB_TC_SEPARATE_BIAS_ROWS", "1")
    for a, b in zip(ops.matmul(r[0], r[1], r[2], r[3], W, bias), plain):
        assert torch.equal(a, b)
    monkeypatch.delenv("FB_TC_SEPARATE_BIAS_ROWS")
    for q in (1.0, 2.0, float("inf")):
        y = ops.matmul_heads_ranges(lw, uw, lb, ub, W, bias, 1, q, eps, 1)
        for a, b in zip(y, ops.matmul(lw, uw, lb, ub, W, bias)):
            assert torch.equal(a, b)
        for a, b in zip(y[4:], ops.concretize(y[0], y[1], y[2], y[3], q, eps, 1)):
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-5)   # (another order of the 128 additions of a norm)
        general = ops.matmul_heads_ranges(lw, lw.clone(), lb, lb.clone(), W, bias, N // 32, q, eps, 1)
        point = ops.matmul_heads_ranges(lw, lw, lb, lb, W, bias, N // 32, q, eps, 1)
        for a, b in zip(point, general):
            assert torch.equal(a, b)
    assert _lib.load().fb_tc_check() == 0


@pytest.mark.parametrize("K,rows", [(128, 304), (512, 1000)])
def test_give_up_path(K, rows):
    """The loads of one k-block of the first thread block left out and every wait limited to about half a millisecond: the block
    drains, frees its tensor memory and returns, the call reports the timeout and the next product is right."""
    from faith_b200 import _lib, ops
    lib = _lib.load()
    lw, uw, lb, ub = _bound(rows, 128, K, 12)
    W, _ = _weight(128, K, 13)
    y = [torch.empty(rows, 128, 128, device=DEV) for _ in range(2)]
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    rc = lib.fb_tc_selftest_timeout(lw.data_ptr(), uw.data_ptr(), W.data_ptr(), y[0].data_ptr(), y[1].data_ptr(), rows * 128, 128, K, 1, 25,
                                    status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 6, lib.fb_status_string(rc)          # FB_ERR_TIMEOUT
    assert int(status.item()) & 4
    assert lib.fb_tc_check() == 0
    _check(ops.matmul(lw, uw, lb, ub, W, None)[:2], lw, uw, W, None, "after the timeout")


@pytest.mark.parametrize("words,positions,p", [(1, [1], float("inf")), (2, [3, 30], 2.0)])
def test_zero_row_blocks_of_the_first_layer_bit_for_bit(words, positions, p):
    import faith_b200
    S = 10
    model = O.make_encoder(4)
    emb = torch.randn(S, 32, 128, generator=torch.Generator().manual_seed(6)).to(DEV)
    ver = faith_b200.EncoderVerifier(model, DEV)
    inst = torch.tensor([[(q + 5 * s) % 32 for q in positions] for s in range(S)], dtype=torch.int32, device=DEV)
    eps_i = torch.full((S,), 1e-3, device=DEV)

    def run():
        a, b = ver.forward(emb, positions, p, 1e-3), ver.forward_instances(emb, inst, p, eps_i)
        return [t.clone() for t in (a[0], a[1], b[0], b[1])]
    fast = run()
    os.environ["FB_ENCODER_NO_ZERO_SKIP"] = "1"
    try:
        plain = run()
    finally:
        del os.environ["FB_ENCODER_NO_ZERO_SKIP"]
    for x, y in zip(fast, plain):
        assert torch.equal(x, y)
    assert bool(torch.isfinite(fast[0]).all()) and bool((fast[0] <= fast[1]).all())
