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
