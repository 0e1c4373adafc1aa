"""The rows of candidates that the grad-h walk records for its passes: lengths
whose squares leave FP32, and smoothing lengths far larger than the cloud,
against the oracle."""
import numpy as np
import pytest

from helpers import case, lists_equal, params, rel_rows, run_pipeline
from oracle.oracle import Oracle
from seren_b200 import ics

pytestmark = pytest.mark.gpu


def _compare(ic, first_call, redo_cap=0):
    from seren_b200.gpu import GpuHotPath
    n = ic["parray"].shape[0]
    g, o = GpuHotPath(n, params(ic, redo_cap=redo_cap)), Oracle(n, params(ic))
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


@pytest.mark.parametrize("h_fac", [1.75, 1.85, 2.2])
def test_rows_that_overflow(h_fac):
    """About 240, 280 and 480 candidates per particle: rows of 256 that mostly hold
    them, mostly hold leaves, and hold leaves only."""
    ic = ics.uniform_sphere(n=20011, seed=73, h_fac=h_fac)
    ic["v"] = np.random.Generator(np.random.PCG64(74)).normal(0.0, 0.1, ic["v"].shape)
    _compare(ic, True)


@pytest.mark.parametrize("precision", [0, 1])
def test_rows_that_overflow_are_not_walked_again(precision):
    """In a steady state of more candidates than a row holds a particle's leaves are
    walked once; the evaluation repeats bit for bit, and its FP64 form agrees with
    the oracle."""
    from seren_b200.gpu import GpuHotPath
    ic = ics.uniform_sphere(n=20011, seed=75, h_fac=2.0)
    n = ic["parray"].shape[0]
    out = []
    for _ in range(2):
        g = GpuHotPath(n, params(ic, precision=precision))
        g.upload(ic["parray"], ic["v"], ic["sound"] ** 2)
        g.force_step(first_call=True)
        g.force_step()
        counts = g.last_step_stats()[2]
        out.append(g.download())
        g.close()
        assert counts[15] > n // 2                       # most rows overflow
        assert counts[3] < 1.1 * n                       # grad-h walks
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
    if precision == 0:
        o = Oracle(n, params(ic))
        p, perm = o.tree_update(ic["parray"])
        s = o.sph_update(p, ic["v"][perm], first_call=True)
        p2, perm2 = o.tree_update(s["parray"])
        s2 = o.sph_update(p2, ic["v"][perm][perm2])
        o.close()
        assert rel_rows(out[0]["rho"], s2["rho"]).max() < 1e-10


@pytest.mark.parametrize("redo_cap", [60, 300])
def test_redo_rounds(redo_cap):
    """Walks that outgrow the redo kernel's first buffers (half of redo_cap) go on in
    its second round when they are more than 1024, and those that outgrow these in
    the whole-GPU rounds."""
    from seren_b200.gpu import GpuHotPath
    ic = case("clumps12k")
    _compare(ic, True, redo_cap)
    n = ic["parray"].shape[0]
    wide = []
    for cap in (redo_cap // 2, redo_cap):
        g = GpuHotPath(n, params(ic, redo_cap=cap))
        g.upload(ic["parray"], ic["v"], ic["sound"] ** 2)
        g.force_step(first_call=True)
        wide.append(g.last_step_stats()[2][8])
        g.close()
    assert wide[0] > 1024                                # outgrow the first buffers
    assert 0 < wide[1] < wide[0]
