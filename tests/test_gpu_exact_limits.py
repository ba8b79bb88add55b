"""Inputs on which the FP64 winding number without all pairs (csrc/wn_exact.cu) could cost
more than the all-pairs kernels that it stands in for: the same values as theirs (bar: the
plain path's 1e-12 per query), at a bounded cost."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from igl import autograd as wa, synthetic  # noqa: E402

pytestmark = pytest.mark.gpu


def _tensors(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in arrays]


def _ms(f):
    times = []
    for _ in range(8):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        f()
        e[1].record()
        torch.cuda.synchronize()
        times.append(e[0].elapsed_time(e[1]))
    return float(np.median(times[2:]))


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("axes", [[0], [1, 2], [0, 1, 2]])
def test_queries_that_are_not_finite(bad, axes):
    """NaN from both paths; none of them is summed over all pairs (half of 65,536 queries:
    64 ms instead of 0.5)."""
    V, F = synthetic.bumpy_icosphere(5, seed=2)
    O = synthetic.mixed_queries(V, F, 20000, seed=3)
    Q = O.copy()
    Q[::2, axes] = bad
    Vt, Ft, Ot, Qt = _tensors(V, F, O, Q)
    tri, ld, nf = wa.triangle_soa(Vt, Ft)
    got, ref = wa.forward_exact(tri, ld, nf, Qt), wa.forward_fp64(tri, ld, nf, Qt)
    assert bool(torch.isnan(ref[::2]).all()) and bool(torch.isnan(got[::2]).all())
    assert float((got - ref)[1::2].abs().max()) <= 1e-12
    assert (_ms(lambda: wa.forward_exact(tri, ld, nf, Qt))
            < 3 * _ms(lambda: wa.forward_exact(tri, ld, nf, Ot)))
