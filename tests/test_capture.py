"""Force calls large enough to make the each-pair-once force's scratch (2^30
pairs of slots) beside and inside a stream capture: the first such call leaves a
capture of another stream whole, may itself be captured, and gives the bits that
it gives without any.
"""
import numpy as np
import pytest
import torch

from hermite_b200 import Gravity
from inputs import make_records

pytestmark = pytest.mark.gpu
EPS2 = (1.0 / 256) ** 2
N = 32768                       # N * N = 2^30


@pytest.fixture(scope="module")
def plain():
    rec = make_records(4, N, seed=91)
    with Gravity(4, N) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        return rec, g.calc_force_on_first_nact(N, EPS2)


def test_first_large_call_beside_a_capture(plain):
    rec, want = plain
    x = torch.ones(1000, device="cuda")
    with Gravity(4, N) as g:
        g.set_jp_records(rec)
        g.predict_all(0.0)
        g.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, capture_error_mode="global"):
            x.add_(1.0)
            g.force_device(N, EPS2)         # on the context's own stream
        got = g.download_forces(N)
        graph.replay()
        torch.cuda.synchronize()
    assert torch.all(x == 2.0)
    assert np.array_equal(got, want)


def test_first_large_call_captured(plain):
    rec, want = plain
    s = torch.cuda.Stream()
    with Gravity(4, N) as g:
        g.set_stream(s.cuda_stream)
        g.set_jp_records(rec)
        g.predict_all(0.0)
        g.predict_pass()                    # not of the graph
        g.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            g.force_device(N, EPS2)
        with torch.cuda.stream(s):
            graph.replay()
        got = g.download_forces(N)
        again = g.calc_force_on_first_nact(N, EPS2)
        del graph
        g.set_stream(None)
    assert np.array_equal(got, want)
    assert np.array_equal(again, want)
