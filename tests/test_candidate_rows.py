"""The rows of candidates that the grad-h walk records for its passes: lengths
whose squares leave FP32, and smoothing lengths far larger than the cloud,
against the oracle."""
import numpy as np
import pytest

from helpers import lists_equal, params, rel_rows, run_pipeline
from oracle.oracle import Oracle
from seren_b200 import ics

pytestmark = pytest.mark.gpu


def _compare(ic, first_call):
    from seren_b200.gpu import GpuHotPath
    n = ic["parray"].shape[0]
    g, o = GpuHotPath(n, params(ic)), Oracle(n, params(ic))
    rg, ro = run_pipeline(g, ic, first_call), run_pipeline(o, ic, first_call)
    limit = g.params.pp_limit
    g.close()
    o.close()
    assert np.array_equal(rg["perm"], ro["perm"])
    sg, so = rg["sph"], ro["sph"]
    assert lists_equal(sg["pptot"], sg["pplist"], so["pptot"], so["pplist"], limit)
    # FP64 sums of some hundred terms in another order
    for k in ("rho", "omega"):
        assert rel_rows(sg[k], so[k]).max() < 1e-11, k
    assert rel_rows(sg["parray"][:, 4:6], so["parray"][:, 4:6]).max() < 1e-11
    assert rel_rows(rg["a"], ro["a"]).max() < 1e-9
    assert rel_rows(rg["gpot"], ro["gpot"]).max() < 1e-11


@pytest.mark.parametrize("first_call", [True, False])
@pytest.mark.parametrize("unit", [1.0e20, 1.0e-8])
@pytest.mark.parametrize("n", [203, 5003])
def test_lengths_of_any_size(n, unit, first_call):
    ic = ics.uniform_sphere(n=n, seed=71)
    ic["parray"][:, [0, 1, 2, 4]] *= unit
    ic["parray"][:, 3] *= unit ** 3                    # the density stays as it is
    _compare(ic, first_call)


@pytest.mark.parametrize("h", [4.0, 1.0e20])
@pytest.mark.parametrize("n", [203, 1003])
def test_smoothing_lengths_beyond_the_cloud(n, h):
    """Every particle is a candidate of every other: 202 fit a row, 1002 do not."""
    ic = ics.uniform_sphere(n=n, seed=72)
    ic["parray"][:, 4] = h
    _compare(ic, False)
