"""Uploads and the kernels that read them share a stream. cudaMemcpy from pageable host
memory may return before the data have reached the device, and the library's own stream is
a non-blocking one, which does not wait for the legacy stream that cudaMemcpy uses."""

import os
import re

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "mojo-libigl_b200", "csrc")


def _function(source: str, name: str) -> str:
    """The body of the function `name` (from its definition to the closing brace)."""
    start = re.search(r"^[\w\s\*]*\b" + name + r"\([^;{]*\)\s*\{", source, re.M)
    assert start, name
    end = source.index("\n}\n", start.end())
    return source[start.end():end]


def test_tree_uploads_are_ordered_before_its_kernels():
    with open(os.path.join(CSRC, "wn_capi.cu")) as f:
        body = _function(f.read(), "wn_aabb_create")
    assert "aabb_discs(" in body  # launches kernels of its own
    assert not re.search(r"\bcudaMemcpy\(|\bcudaMemset\(", body)
    assert "cudaStreamSynchronize(" in body  # the host arrays end with the call


@pytest.mark.parametrize("name", ["context", "wn_mixed_stats", "fwn_upload", "wn_batch_create"])
def test_other_uploads_are_waited_for(name):
    with open(os.path.join(CSRC, "wn_capi.cu")) as f:
        body = _function(f.read(), name)
    copies = list(re.finditer(r"\bcudaMemcpy\(|\bcudaMemset\(|batch_edges_create\(", body))
    assert copies and "uploads_done()" in body[copies[-1].end():]


@pytest.mark.gpu
def test_trees_made_one_after_another():
    """Trees with and without thin faces in turn, each checked against the host's walk."""
    torch = pytest.importorskip("torch")
    import igl
    from igl import distance, synthetic

    V, F = synthetic.bumpy_icosphere(6, seed=3)
    thin = np.concatenate([F, np.stack([F[:, 0], F[:, 0], F[:, 1]], 1)[:1]])
    P = np.concatenate([synthetic.mixed_queries(V, F, 500, seed=1, near_sigma=1e-3), V[:50]])
    expected = []
    for faces in (F, thin):
        host = igl.AABB()
        host.init(V, faces)
        expected.append(host.squared_distance(V, faces, P))
    side = torch.cuda.Stream()  # non-blocking: ordered after the upload by the call alone
    p = torch.from_numpy(P).cuda()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for i in range(12):
            tree = distance.DeviceAABB(V, (F, thin)[i % 2])
            for a, b in zip(tree.query(p), expected[i % 2]):
                assert a.cpu().numpy().tobytes() == np.asarray(b).tobytes()
            tree.close()


def test_host_forward_uploads_its_inputs_once():
    """Also where the path without all pairs declines and an all-pairs kernel runs."""
    with open(os.path.join(CSRC, "wn_capi.cu")) as f:
        body = _function(f.read(), "forward_fp64_host")
    assert len(re.findall(r"cudaMemcpy2DAsync\(", body)) == 1
    assert len(re.findall(r"cudaMemcpyHostToDevice", body)) == 2  # the soup and the queries
