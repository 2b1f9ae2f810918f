"""The cell walk (neighbor walk 2 over cells of one kernel reach) where its
staging changes form: cells with more nodes than one, two and four registers
per lane hold, cells it leaves unordered, windows beyond the staging area and
beyond the tested candidates, nodes in no order.  The ConnectivityMap is
integer work: every entry equals the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _clump(pkg, clump, seed, periodic, vary):
    """A 10^3 lattice in the unit cube (reach 0.16: about 4 nodes per cell) with `clump` nodes within 0.02 of a point."""
    gen, abi = pkg.generators, pkg.abi
    ns = gen.kelvin_helmholtz(nx=10, ny=10, nz=10, jitter=0.2, seed=seed)
    rng = np.random.default_rng(seed)
    pos = np.concatenate([ns.pos, np.array([0.41, 0.97, 0.52]) + rng.uniform(-0.02, 0.02, (clump, 3))])
    n = pos.shape[0]
    h = 0.08 * (rng.uniform(0.9, 1.0, n) if vary else np.ones(n))
    H = np.zeros((n, 6))
    H[:, [0, 3, 5]] = 1.0 / h[:, None]
    perm = rng.permutation(n)
    full = gen.NodeSet(pos[perm], np.zeros((n, 3)), np.full(n, 1.0 / n), np.ones(n), np.ones(n), H[perm], ns.dx)
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, periodic=periodic, max_neighbors=2048)
    return full, cfg


# 20: one register per lane; 50, 100: two and four; 140: a cell left unordered; 800: the 27 cells still fit the
# staging area, 1100: more than a ballot word per lane; 1700: more than the staging area
@pytest.mark.parametrize("clump", [20, 50, 100, 140, 800, 1100, 1700])
@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("periodic,vary", [((1, 1, 1), False), ((1, 0, 1), True)])
def test_clumped_cells(gpu_lib, pkg, oracle_mod, clump, passes, periodic, vary):
    ns, cfg = _clump(pkg, clump, 7 + clump, periodic, vary)
    g = pkg.SPHHydro(cfg, ns)
    g.set_schedule("neighbor walk", 2)
    g.set_schedule("neighbor passes", passes)
    o = oracle_mod.OracleProblem(cfg, ns)
    o.build_neighbors()
    oo, on, orr = o.connectivity()
    for _ in range(2):                       # the second build is planned from the first
        g.build_neighbors()
        go, gn, gr = g.connectivity()
        assert np.array_equal(go, oo) and np.array_equal(gn, on) and np.array_equal(gr, orr)
        assert g.num_pairs() == o.num_pairs()
