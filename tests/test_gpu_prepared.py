"""forward_fp64_prepared: FP64 pairs over a mesh prepared for the call. Nothing in the package
calls it any more (the streaming kernel is the faster one), and callers may."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from igl import autograd as wa, synthetic  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level, queries", [(2, 1), (3, 1000), (5, 4097)])
def test_against_the_streaming_kernel(level, queries):
    V, F = synthetic.bumpy_icosphere(level, seed=level)
    F = synthetic.delete_faces(F, 0.05, seed=1)
    O = synthetic.mixed_queries(V, F, queries, seed=2)
    Vt, Ft, Ot = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (V, F, O))
    tri, ld, nf = wa.triangle_soa(Vt, Ft)
    w = wa.forward_fp64_prepared(tri, ld, nf, Ot)
    assert float((w - wa.forward_fp64(tri, ld, nf, Ot)).abs().max()) <= 1e-12
