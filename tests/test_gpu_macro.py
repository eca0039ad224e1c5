"""GPU tests of the field getter (fetch_macro in csrc/capi.cu), whose host threads copy the moments in
blocks of 8192 fluid nodes. The fields are copies: tolerance 0 throughout."""
import numpy as np
import pytest

import piks3d_b200 as pk
from conftest import base_params
from piks3d_b200 import images

pytestmark = pytest.mark.gpu

STREAM_LEGACY, STREAM_PER_THREAD = 1, 2   # cudaStreamLegacy, cudaStreamPerThread


def _fields(img, p, stream, wait):
    with pk.Solver(p, device=0) as s:
        if stream:
            s.set_stream(stream)
        s.setup_physical_grid(img)
        s.iterate(60)
        if wait:
            s.synchronize()
        return s.get_macro()


@pytest.mark.parametrize("edge", [20, 33, 48])
@pytest.mark.parametrize("stream", [None, STREAM_LEGACY, STREAM_PER_THREAD])
def test_fields_wait_for_the_iterations_of_the_callers_stream(edge, stream):
    """Boxes of one block, a few and a dozen: the fields right after the iterations were enqueued
    equal those of a context that waited for them first. cudaStreamPerThread names another stream
    in every host thread."""
    img = images.sphere_pack(edge, 0.6, 2.0, 4.0, seed=3)
    p = base_params(edge, Nc_fundamental=4, Kn=0.8, wallExtOrder=1)
    want = _fields(img, p, None, True)
    got = _fields(img, p, stream, False)
    assert any(np.any(w) for w in want)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("edge", [16, 40])
def test_fields_are_the_same_on_every_call(edge):
    """The first call of a context stages a small box in pageable memory, later ones in pinned."""
    img = images.sphere_pack(edge, 0.7, 2.0, 4.0, seed=6)
    with pk.Solver(base_params(edge, wallExtOrder=1), device=0) as s:
        s.setup_physical_grid(img)
        s.iterate(12)
        first, rest = s.get_macro(), [s.get_macro() for _ in range(3)]
        assert any(np.any(f) for f in first)
        for got in rest:
            for a, b in zip(got, first):
                assert np.array_equal(a, b)
