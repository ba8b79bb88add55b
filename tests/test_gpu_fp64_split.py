"""The streaming FP64 forward at the edges of its shapes (queries per CTA, faces per tile
and step, odd ends) against the library's host path. Bar 1e-12: at most 1,000 faces, each
term within a few 1e-16 of its angle. Queries on vertices, sides and faces take the
bit-identical terms in both, so no half turn may differ; scaling by a power of two
changes no term but takes all of them out of the cheaper terms' range."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import igl  # noqa: E402
from igl import _lib, autograd as wa  # noqa: E402

pytestmark = pytest.mark.gpu


def _soup(nf, seed):
    """Faces of a bumpy sphere, thin, repeated and degenerate ones among them."""
    V, F = igl.synthetic.bumpy_icosphere(3, seed=seed)
    F = F[np.random.default_rng(seed).permutation(len(F))[:nf]].copy()
    if nf > 8:
        F[3], F[5] = F[2], F[4][[0, 0, 1]]
    return V, F


def _queries(V, F, nq, seed):
    rng = np.random.default_rng(seed)
    O = rng.uniform(-1.3, 1.3, size=(nq, 3))
    if len(F):
        f = V[F[rng.integers(0, len(F), size=nq)]]
        O[1::5] = f[1::5, 0]
        O[2::5] = 0.5 * (f[2::5, 0] + f[2::5, 1])
        O[3::5] = f[3::5].mean(1) + rng.normal(scale=1e-9, size=(len(O[3::5]), 3))
    return O


def _device(V, F, O, mode):
    tri, ld, nf = wa.triangle_soa(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda())
    q = torch.from_numpy(O).cuda()
    w = torch.full((len(O),), np.nan, dtype=torch.float64, device="cuda")
    assert not _lib.lib().wn_forward_fp64_device(
        tri.data_ptr(), ld, q.data_ptr(), w.data_ptr(), nf, len(O), mode,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return w.cpu().numpy()


@pytest.mark.parametrize("nf", [0, 1, 2, 63, 64, 65, 127, 129, 1000])
@pytest.mark.parametrize("nq", [1, 3, 4, 5, 80, 84, 85, 128, 129, 168, 169, 257, 1025])
def test_shapes(nf, nq):
    V, F = _soup(nf, 11)
    O = _queries(V, F, nq, nf + nq)
    want = igl.winding_number(V, F, O, device="cpu")
    for mode in (0, 1):
        assert np.abs(_device(V, F, O, mode) - want).max() <= 1e-12


@pytest.mark.parametrize("nq", [40, 600])
@pytest.mark.parametrize("scale", [2.0**-260, 2.0**-98, 1.0, 2.0**98, 2.0**260])
def test_scales(scale, nq):
    V, F = _soup(1000, 12)
    O = _queries(V, F, nq, 13)
    want = igl.winding_number(V, F, O, device="cpu")
    assert np.abs(_device(V * scale, F, O * scale, 0) - want).max() <= 1e-12


def test_many_faces_for_few_queries():
    """A few-query CTA's threads take several faces each, in several splits."""
    V, F = igl.synthetic.terrain_grid(350)
    O = _queries(V, F, 5, 14)
    O[0] = V.mean(0)  # 243,602 faces: the bar grows with the root of their number
    want = igl.winding_number(V, F, O, device="cpu")
    assert np.abs(_device(V, F, O, 0) - want).max() <= 1e-11
