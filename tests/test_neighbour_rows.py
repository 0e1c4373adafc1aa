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
@pytest.mark.parametrize("kind,n,pp_limit", [
    ("plummer", 20001, None), ("disc", 5003, None), ("plummer", 20001, 60), ("disc", 5003, 60)])
def test_force_step_repeats_bit_for_bit(kind, n, pp_limit, precision):
    """The same input gives the same bits, and in FP64 the oracle's numbers; with
    scatter parts of more and fewer than 16 entries, redone particles, and rows
    that overflow pp_limit."""
    from seren_b200.gpu import GpuHotPath
    ic = (ics.plummer if kind == "plummer" else ics.protostellar_disc)(n=n, seed=61)
    ic["sound"] = np.full(n, 0.1)
    prm = params(ic, precision=precision)
    if pp_limit:
        prm.pp_limit = pp_limit
    first = None
    for _ in range(3):
        g = GpuHotPath(n, prm)
        out = g.force_step_io(ic["parray"], ic["v"], ic["sound"] ** 2, first_call=True)
        assert g.last_step_stats()[2][15] > 0               # particles redone
        out = g.force_step_io(out["parray"], out["v"], out["csq"])
        g.close()
        if first is None:
            first = out
        for k in first:
            assert np.array_equal(first[k], out[k]), k
    # the oracle's second evaluation, and what its lists hold
    o = Oracle(n, params(ic))
    p, perm = o.tree_update(ic["parray"])
    s = o.sph_update(p, ic["v"][perm], first_call=True)
    v = ic["v"][perm]
    p, perm = o.tree_update(s["parray"])
    v = v[perm]
    s = o.sph_update(p, v)
    sound = np.full(n, 0.1)
    a, _ = o.grav_forces(o.hydro_forces(sound * sound * s["rho"], sound))
    o.close()
    p, tot = s["parray"], s["pptot"]
    if kind == "plummer" or pp_limit:
        assert (tot > prm.pp_limit).any()                   # rows without a list
    short = np.flatnonzero(tot <= prm.pp_limit)
    scatter = np.zeros(n, int)                              # neighbours beyond a row's own 2h
    for i in short:
        d = p[s["pplist"][i, :tot[i]], 0:3] - p[i, 0:3]
        scatter[i] = np.count_nonzero((d * d).sum(axis=1) > 4.0 * p[i, 4] ** 2)
    assert (scatter > 16).any() and ((scatter > 0) & (scatter <= 16)).any()
    if precision == 0:
        # FP64 sums of some hundred terms in another order
        assert rel_rows(first["rho"], s["rho"]).max() < 1e-11
        assert rel_rows(first["a"], a).max() < 1e-9


# (100003 particles: the walks' scratch takes the 1000 sinks in two rounds)
@pytest.mark.parametrize("n,nsink", [(37, 1), (5000, 3), (5000, 200), (100003, 1000)])
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
