"""Team sizes chosen by the library.  Ensembles: powers of two of at most 512 slots
per CTA, nine in place of eight, which fill the GPU where many clusters are of one size (a CTA per 384
slots took up to 1.8 times as long there), and the same results as teams of that
size asked for."""
import numpy as np
import pytest

from hermite_b200 import Ensemble, Gravity
from hermite_b200.ic import plummer, records

pytestmark = pytest.mark.gpu


def test_automatic_sizes():
    sizes = [1, 512, 513, 1024, 1025, 2048, 2049, 4096, 4097, 8000]
    with Ensemble(4, sizes, "fp64") as e:
        assert [e.cluster_engine(c) for c in range(len(sizes))] == \
            [("team", k) for k in (1, 1, 2, 2, 4, 4, 9, 9, 16, 16)]


def test_same_as_asked_for():
    n, out = 1500, []
    for engine, ctas in (("auto", 0), ("team", 4)):
        with Ensemble(4, [n, n], "fp64") as e:
            e.set_engine(engine, ctas)
            for c in range(2):
                e.set_cluster(c, records(plummer(n, c), 4), (4 / n) ** 2)
            e.init(0.0, 0.02, 0.005, 1 / 128)
            e.run(1 / 128)
            out.append([e.get_cluster(c) for c in range(2)])
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("n,ctas", [(1, 1), (33, 2), (512, 16), (513, 9), (700, 11), (1024, 16), (1025, 11), (2560, 16)])
def test_single_system(n, ctas):
    """No more CTAs than the chunks per CTA of the largest team call for."""
    with Gravity(8, n) as g:
        assert g.engine() == ("team", ctas)
