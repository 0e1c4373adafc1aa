"""Rows whose order depends on atomics until they are sorted, and walks spread
over a block: results that repeat bit for bit, and many sinks against the
oracle."""
import numpy as np
import pytest

from helpers import params, rel_rows
from oracle.oracle import Oracle
from seren_b200 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind,n", [("plummer", 20001), ("disc", 5003)])
def test_force_step_repeats_bit_for_bit(kind, n, precision):
    """Scatter parts of more and fewer than 16 entries, overflowed rows, redone
    particles: the same input gives the same bits."""
    from seren_b200.gpu import GpuHotPath
    ic = (ics.plummer if kind == "plummer" else ics.protostellar_disc)(n=n, seed=61)
    first = None
    for _ in range(3):
        g = GpuHotPath(n, params(ic, precision=precision))
        out = g.force_step_io(ic["parray"], ic["v"], ic["sound"] ** 2, first_call=True)
        out = g.force_step_io(out["parray"], out["v"], out["csq"])
        g.close()
        if first is None:
            first = out
        for k in first:
            assert np.array_equal(first[k], out[k]), k


@pytest.mark.parametrize("n,nsink", [(37, 1), (5000, 3), (5000, 200)])
def test_sink_forces_of_many_sinks(n, nsink):
    from seren_b200.gpu import GpuHotPath
    ic = ics.plummer(n=n, seed=62)
    rng = np.random.Generator(np.random.PCG64(63))
    sinks = np.zeros((nsink, 5))
    sinks[:, 0:3] = rng.normal(0.0, 1.0, (nsink, 3))
    sinks[:, 3] = rng.uniform(0.01, 0.1, nsink)
    sinks[:, 4] = rng.uniform(0.01, 0.5, nsink)
    g, o = GpuHotPath(n, params(ic)), Oracle(n, params(ic))
    g.tree_update(ic["parray"])
    o.tree_update(ic["parray"])
    ag, pg = g.sink_forces(sinks)
    ao, po = o.sink_forces(sinks)
    g.close()
    o.close()
    # FP64 sums of up to n terms in another order
    assert rel_rows(ag, ao).max() < 1e-11 and rel_rows(pg, po).max() < 1e-12


@pytest.mark.parametrize("precision", [0, 1])
def test_hydro_after_a_restock(precision):
    """Rows over pp_limit are searched on the fly, by the cells' search ranges of the
    last sph_update: a restock of the same particles leaves those as they are.
    (Smoothing lengths that differ from cell to cell: many neighbours are found by
    the scatter test only.)"""
    from seren_b200.gpu import GpuHotPath
    n = 4001
    ic = ics.plummer(n=n, seed=64)
    prm = params(ic, precision=precision)
    prm.pp_limit = 30
    g = GpuHotPath(n, prm)
    p, perm = g.tree_update(ic["parray"])
    s = g.sph_update(p, ic["v"][perm], first_call=True)
    assert (s["pptot"] > prm.pp_limit).mean() > 0.5
    sound = np.full(n, 0.1)
    press = sound * sound * s["rho"]
    a = g.hydro_forces(press, sound)
    g.tree_update(s["parray"], do_build=False)
    again = g.hydro_forces(press, sound)
    g.close()
    assert np.array_equal(a, again)
