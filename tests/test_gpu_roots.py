"""The reciprocal square root and reciprocal of the cheaper FP64 pair terms (wn_common.cuh):
the hardware's approximation and one third-order step. The step leaves 5 e^3 / 16 and e^3 of
the approximation's relative error e < 2^-18, so what remains is the rounding of the last two
operations: at most one unit of 2^-53 for the result and half of one for the correction, 2^-52
in all. Compared in 64-bit mantissas on the host, and with CUDA's own functions."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from igl import _lib, autograd as wa  # noqa: E402

pytestmark = pytest.mark.gpu


def _roots(x):
    t = torch.from_numpy(x).cuda()
    a, b = torch.empty_like(t), torch.empty_like(t)
    assert _lib.lib().wn_probe_roots_device(t.data_ptr(), len(x), a.data_ptr(), b.data_ptr(),
                                            wa._stream()) == 0
    return t, a, b


@pytest.mark.parametrize("low, high", [(-600, 600), (-2, 2), (-1000, -900), (900, 1000)])
def test_error(low, high):
    rng = np.random.default_rng(low + 2000)
    x = np.ldexp(rng.uniform(0.5, 1.0, 1 << 20), rng.integers(low, high + 1, 1 << 20))
    x[:200] = np.ldexp(1.0 + np.arange(200) * 2.0 ** -52, low)  # just above a power of two
    x[200:400] = np.ldexp(1.0 - np.arange(200) * 2.0 ** -53, high)
    t, a, b = _roots(x)
    exact = np.longdouble(x)
    assert np.finfo(np.longdouble).nmant >= 63
    for got, want, cuda in ((a, 1 / np.sqrt(exact), torch.rsqrt(t)), (b, 1 / exact, 1 / t)):
        error = np.abs(got.cpu().numpy() / want - 1).max()
        assert error <= 2.0 ** -52
        assert float((got / cuda - 1).abs().max()) <= 2.0 ** -51


def test_what_has_no_finite_root_gives_none():
    x = np.array([0.0, -0.0, np.inf, np.nan, 5e-324, 1e-310])
    _, a, b = _roots(x)
    assert not np.isfinite(a.cpu().numpy()).any()
    assert not np.isfinite(b.cpu().numpy()).any()
    assert not np.isfinite(_roots(np.array([-1.0, -1e300]))[1].cpu().numpy()).any()
