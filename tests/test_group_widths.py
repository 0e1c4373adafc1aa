"""Group widths of the gravity walk (32, 16, 8 or 4 particles per warp, chosen
by the cloud's size): each width at the edge of its range against the oracle,
and clouds of different widths in one forest against the same clouds alone."""
import numpy as np
import pytest

from helpers import params, rel_rows, rel_scaled
from oracle.oracle import Oracle
from seren_b200 import ics

pytestmark = pytest.mark.gpu


def _gravity(hp, ic):
    p, perm = hp.tree_update(ic["parray"])
    return hp.grav_forces(), perm


@pytest.mark.parametrize("n", [33, 4096, 4097, 16384, 16385, 65537])
def test_gravity_at_the_width_edges(n):
    from seren_b200.gpu import GpuHotPath
    ic = ics.plummer(n=n, seed=31)
    o = Oracle(n, params(ic))
    (ao, po), permo = _gravity(o, ic)
    for precision in (0, 1):
        g = GpuHotPath(n, params(ic, precision=precision))
        (ag, pg), permg = _gravity(g, ic)
        g.close()
        assert np.array_equal(permg, permo)
        if precision == 0:
            # sums of about 1000 terms of a few 2^-52 each
            assert rel_rows(ag, ao).max() < 1e-11 and rel_rows(pg, po).max() < 1e-12
        else:
            # 32-bit terms: a few 2^-24 of the largest contributions, and a pair that the
            # 32-bit separation puts into the next bin of the kernel (2e-4 h wide)
            # changes its term by up to 1e-4, of a sum of at least 32
            assert rel_scaled(ag, ao) < 1e-5 and rel_rows(pg, po).max() < 1e-5
    o.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_forest_of_clouds_of_every_width(precision):
    from seren_b200.gpu import GpuHotPath
    ns = [70001, 130, 4500, 17003, 4096]
    clouds = [ics.uniform_sphere(n=n, seed=40 + k) for k, n in enumerate(ns)]
    g = GpuHotPath(sum(ns), params(clouds[0], precision=precision))
    g.upload(np.vstack([c["parray"] for c in clouds]), np.vstack([c["v"] for c in clouds]),
             np.concatenate([c["sound"] ** 2 for c in clouds]))
    g.set_clouds(ns)
    g.force_step(first_call=True)
    st = g.download()
    g.close()
    off = 0
    for ic, n in zip(clouds, ns):
        one = GpuHotPath(n, params(ic, precision=precision))
        one.upload(ic["parray"], ic["v"], ic["sound"] ** 2)
        one.force_step(first_call=True)
        s1 = one.download()
        one.close()
        for k in ("parray", "rho", "omega", "a", "gpot"):
            assert np.array_equal(st[k][off:off + n], s1[k]), (n, k)
        off += n
