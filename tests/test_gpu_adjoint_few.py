"""The FP64 adjoint of few boundary edges (csrc/wn_adjoint.cu), around the number from which a
thread takes four of them instead of two, against the variant with the CUDA library's roots
and division. Both round every term to a few units of 2^-53; a gradient entry adds up to
2,049 (dL/dq) or 20,001 (an edge's ends) of them, whose sizes sum to at most 1e3 times its
bar's unit here: 1e-12 of the largest entry."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from igl import _lib, autograd as wa  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edges", [1, 3, 127, 128, 129, 255, 256, 257, 511, 513, 2049])
@pytest.mark.parametrize("queries", [1, 63, 65, 20001])
def test_edges(edges, queries):
    rng = np.random.default_rng(edges)
    P = rng.uniform(-1, 1, size=(edges, 3))
    E = np.concatenate([P.T, (P + 0.1 * rng.normal(size=P.shape)).T,
                        rng.choice([-2.0, -1.0, 1.0, 3.0], size=(1, edges))])
    O = rng.normal(size=(queries, 3))
    O *= (2.5 + np.abs(rng.normal(size=(queries, 1)))) / np.linalg.norm(O, axis=1, keepdims=True)
    e, q, g = (torch.from_numpy(np.ascontiguousarray(x)).cuda()
               for x in (E, O, rng.normal(size=queries)))
    handle = _lib.lib()
    out = []
    for adjoint in (handle.wn_backward_edges_open_device, handle.wn_backward_edges_device):
        dq, de = torch.empty_like(q), torch.empty(6, edges, dtype=torch.float64, device="cuda")
        assert adjoint(e.data_ptr(), edges, edges, q.data_ptr(), queries, g.data_ptr(),
                       dq.data_ptr(), de.data_ptr(), wa._stream()) == 0
        out.append((dq, de))
    for a, b in zip(*out):
        assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max())
