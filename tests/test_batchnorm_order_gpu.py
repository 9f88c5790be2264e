"""Batch norm over row counts at the edges of its blocks and trips (the backward pass goes through them from the end)."""
import pytest
import torch

from tnn_b200.ops import _lib, raw

pytestmark = pytest.mark.gpu


# rows: below one trip, one row past a trip, ragged blocks, many trips
@pytest.mark.parametrize("M,C", [(1, 8), (3, 24), (1023, 8), (1025, 8), (33, 256), (12545, 264), (70001, 64), (401, 2048)])
@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("resid", [False, True])
def test_rows_are_each_written_once(M, C, relu, resid):
    g = torch.Generator(device="cuda").manual_seed(M + C)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    x, res, dy = rnd(M, C), rnd(M, C) if resid else None, rnd(M, C)
    gamma, beta = 1 + 0.1 * rnd(C), 0.1 * rnd(C)
    rm, rv = torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
    y, mean, rstd = raw.batchnorm_fwd_train(x, gamma, beta, rm, rv, 1e-5, 0.1, relu, resid=res)
    xd = x.double()
    mu, var = xd.mean(0), xd.var(0, unbiased=False)
    pre = (xd - mu) * (var + 1e-5).rsqrt() * gamma.double() + beta.double()
    ref = pre + (res.double() if resid else 0)
    ref = ref.clamp_min(0) if relu else ref
    # one rounding of the result and, with a residual, one of the normalised value; fp32 statistics
    bound = 2.0 ** -8 * (ref.abs() + pre.abs()) + 2.0 ** -14 * (1 + (var + 1e-5).rsqrt() * xd.abs().max())
    assert bool(((y.double() - ref).abs() <= bound).all())
    yi = raw.batchnorm_infer(x, gamma, beta, rm, rv, 1e-5, relu, resid=res)
    pre = (xd - rm.double()) * (rv.double() + 1e-5).rsqrt() * gamma.double() + beta.double()
    ref = pre + (res.double() if resid else 0)
    ref = ref.clamp_min(0) if relu else ref
    assert bool(((yi.double() - ref).abs() <= 2.0 ** -8 * (ref.abs() + pre.abs()) + 2.0 ** -14).all())
    if resid:
        return
    dg, db = torch.zeros(C, device="cuda"), torch.zeros(C, device="cuda")
    dx = raw.batchnorm_bwd(dy, x, y, mean, rstd, gamma, dg, db, relu)
    _lib.check_status()
    live = (y > 0).double() if relu else 1.0
    gd, rs = dy.double() * live, rstd.double()
    xh = (xd - mean.double()) * rs
    sg, sgx = gd.sum(0), (gd * xh).sum(0)
    rdx = gamma.double() * rs * (gd - sg / M - xh * sgx / M)
    scale = (gamma.double() * rs).abs() * (gd.abs() + gd.abs().mean(0) + xh.abs() * (gd * xh).abs().mean(0))
    assert bool(((dx.double() - rdx).abs() <= 2.0 ** -8 * rdx.abs() + 2.0 ** -18 * scale).all())
