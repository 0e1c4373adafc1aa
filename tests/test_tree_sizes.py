"""The tree build at the sizes where it changes: one-block sort up to 4096
particles, small and large radix tiles (2^19), the sort on the upper digits only
and again on all of them for trees of more than 10 levels, blocks of 256
particles; cells and order bit for bit against the oracle."""
import numpy as np
import pytest

from helpers import deep_clump, params
from oracle.oracle import Oracle
from seren_b200 import ics

pytestmark = pytest.mark.gpu

INTS = ("leaf", "nextcell", "ifopen", "plist", "first_cell", "last_cell")
FLOATS = ("grav_r", "grav_m", "grav_q", "dminsqd", "hydro_r", "rmax")


def _compare(g, o, parray):
    pg, permg = g.tree_update(parray)
    po, permo = o.tree_update(parray)
    assert np.array_equal(permg, permo) and np.array_equal(pg, po)
    tg, to = g.tree_export(), o.tree_export()
    assert tg["ctot"] == to["ctot"] and tg["ltot"] == to["ltot"]
    for k in INTS + FLOATS:
        assert np.array_equal(tg[k], to[k]), k
    return tg["ltot"]


@pytest.mark.parametrize("kind,n", [
    ("sphere", 1), ("sphere", 8), ("sphere", 9), ("sphere", 255), ("sphere", 257),
    ("sphere", 4096), ("sphere", 4097), ("plummer", 4096), ("plummer", 20000),
    ("disc", 60001), ("sphere", 524287), ("sphere", 524289)])
def test_tree_at_the_size_edges(kind, n):
    from seren_b200.gpu import GpuHotPath
    make = {"sphere": ics.uniform_sphere, "plummer": ics.plummer, "disc": ics.protostellar_disc}
    ic = make[kind](n=n, seed=51)
    g, o = GpuHotPath(n, params(ic)), Oracle(n, params(ic))
    _compare(g, o, ic["parray"])
    g.close()
    o.close()


def test_shallow_tree_after_a_deep_one_and_back():
    """The context's choice of sort follows the trees it builds."""
    from seren_b200.gpu import GpuHotPath
    n = 30000
    deep, flat = ics.plummer(n=n, seed=3), ics.uniform_sphere(n=n, seed=4)
    deep["parray"][: n // 2, 0:3] *= 1.0e-3
    g, o = GpuHotPath(n, params(flat)), Oracle(n, params(flat))
    depths = [_compare(g, o, ic["parray"]) for ic in (flat, deep, deep, flat, flat, deep)]
    assert max(depths[1:3]) > 10 and depths[0] <= 10 and depths[3] <= 10
    g.close()
    o.close()


def test_deep_tree_of_many_blocks():
    """24 levels and 80000 particles: the cells are written while other blocks put
    their leaves' particles into input order."""
    from seren_b200.gpu import GpuHotPath
    ic = deep_clump(1.0e-5, n_core=40000, n_halo=40000)
    n = ic["parray"].shape[0]
    g, o = GpuHotPath(n, params(ic)), Oracle(n, params(ic))
    assert _compare(g, o, ic["parray"]) > 21
    g.close()
    o.close()


def test_forest_of_more_roots_than_a_block_takes():
    """1030 clouds: the level of the roots is stocked like any other; some of the
    clouds against the same clouds alone, bit for bit."""
    from seren_b200.gpu import GpuHotPath
    m, ncl = 70, 1030
    kinds = [ics.uniform_sphere(n=m, seed=80 + k) for k in range(5)]
    clouds = [kinds[k % 5] for k in range(ncl)]
    g = GpuHotPath(m * ncl, params(kinds[0]))
    g.upload(np.vstack([c["parray"] for c in clouds]), np.vstack([c["v"] for c in clouds]),
             np.concatenate([c["sound"] ** 2 for c in clouds]))
    g.set_clouds([m] * ncl)
    g.force_step(first_call=True)
    st = g.download()
    g.close()
    for k, ic in enumerate(kinds):
        one = GpuHotPath(m, params(ic))
        one.upload(ic["parray"], ic["v"], ic["sound"] ** 2)
        one.force_step(first_call=True)
        s1 = one.download()
        one.close()
        for c in (k, ncl - 5 + k):
            for name in ("parray", "rho", "omega", "a", "gpot"):
                assert np.array_equal(st[name][c * m:(c + 1) * m], s1[name]), (c, name)
