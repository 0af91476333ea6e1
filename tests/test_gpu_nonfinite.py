"""An infinity or NaN in the input makes those elements of the product non-finite
that the matrix connects it with, and no others, on every path.

The blocked same-spin kernels and the stored Hamiltonian's blocks hold zeros for
strings that do not connect, and zero times an infinity is NaN. The one-string
kernels (codes 22 and 24) hold none and say which elements are finite; those are
equal within 1e-12 (FP64) and 2e-6 (FP32 storage) of the largest. The next
finite product is as before.
"""
import numpy as np
import pytest
import torch

import sbdx
from sbdx import synth

pytestmark = pytest.mark.gpu


def check(got, want, tol):
    got, want = got.reshape(-1), want.reshape(-1)
    f = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), f)
    assert f.any() and not f.all()
    assert np.abs(got[f] - want[f]).max() <= tol * np.abs(want[f]).max()


@pytest.fixture(scope="module", params=[(24, 5, 5, 150, 131), (20, 4, 5, 61, 300)])
def prob(request):
    return synth.random_problem(*request.param, seed=71)


def product(ctx, x):
    s = torch.empty_like(x)
    ctx.sigma_device(sbdx.SBDX_FP64 if x.dtype == torch.float64 else sbdx.SBDX_FP32, x.data_ptr(), s.data_ptr())
    torch.cuda.synchronize()
    return s.double().cpu().numpy()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_blocked_and_stored_products(prob, value):
    C = np.random.default_rng(72).standard_normal(prob.D)
    bad = C.copy()
    bad[(prob.na // 2) * prob.nb + 7] = value
    bad[3 * prob.nb + prob.nb // 3] = value
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        for dtype, plain, tol in ((torch.float64, 22, 1e-12), (torch.float32, 24, 2e-6)):
            x, xb = torch.from_numpy(C).cuda().to(dtype), torch.from_numpy(bad).cuda().to(dtype)
            ctx.set_tuning(plain, 71)
            want = product(ctx, xb)
            ctx.set_tuning(34, 71)
            before = product(ctx, x)
            check(product(ctx, xb), want, tol)
            assert np.array_equal(product(ctx, x), before)
            if dtype == torch.float64:
                a0 = prob.na // 3 // 8 * 8
                rows = torch.empty((prob.na - a0, prob.nb), dtype=dtype, device="cuda")
                ctx.sigma_rows_device(sbdx.SBDX_FP64, xb.data_ptr(), rows.data_ptr(), a0, prob.na)
                torch.cuda.synchronize()
                check(rows.cpu().numpy(), want.reshape(prob.na, prob.nb)[a0:], tol)
                ctx.set_io_chunks(3)
                check(ctx.sigma(bad), want, tol)
                ctx.set_io_chunks(0)
                assert np.array_equal(product(ctx, x), before)
        ctx.build_hamiltonian()
        ctx.set_tuning(22, 71)
        x, xb = torch.from_numpy(C).cuda(), torch.from_numpy(bad).cuda()
        got = product(ctx, xb)
        ctx.release_hamiltonian()
        check(got, product(ctx, xb), 1e-12)
