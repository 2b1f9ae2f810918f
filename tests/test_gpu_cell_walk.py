"""The cell walk (neighbor walk 2 over cells of one kernel reach) where its
staging changes form: cells with more nodes than one, two and four registers
per lane hold, cells it leaves unordered, windows beyond the staging area and
beyond the tested candidates, nodes in no order, any unit of length, crowded
cells that come and go.  The ConnectivityMap is integer work: every entry equals
the oracle's."""
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


# 20: one register per lane in the cells' ordering; 50, 100: two and four; 140 and more: cells left unordered, whose
# windows are all crowded (test_full_windows has the windows that fill the staging area and the ballots)
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


def _same_connectivity(g, o):
    oo, on, orr = o.connectivity()
    go, gn, gr = g.connectivity()
    assert np.array_equal(go, oo) and np.array_equal(gn, on) and np.array_equal(gr, orr)
    assert g.num_pairs() == o.num_pairs()


# 1e-24 and 1e21: squares of lengths vanish or overflow in FP32; 1e19: some of them do
@pytest.mark.parametrize("unit", [1.0e-24, 1.0, 1.0e19, 1.0e21])
@pytest.mark.parametrize("form", ["pre-test", "exact", "spread"])
@pytest.mark.parametrize("walk,cells", [(2, 1), (2, 2), (1, 1), (1, 2)])
def test_units_of_length(gpu_lib, pkg, oracle_mod, unit, form, walk, cells):
    """The FP32 tests of the walks decide nothing wrongly in any unit of length,
    with the pre-test, without it, and with smoothing scales more than 100 apart
    (where it is off)."""
    gen, abi = pkg.generators, pkg.abi
    ns, _ = _clump(pkg, 50, 3, (1, 0, 1), True)
    if form == "spread":
        ns.H[::3, [0, 3, 5]] *= 150.0
    big = gen.NodeSet(ns.pos * unit, ns.vel, ns.mass, ns.rho, ns.eps, ns.H / unit, ns.dx * unit)
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, periodic=(1, 0, 1), max_neighbors=2048, xmax=(unit,) * 3)
    g, o = pkg.SPHHydro(cfg, big), oracle_mod.OracleProblem(cfg, big)
    g.set_schedule("neighbor walk", walk)
    g.set_schedule("neighbor cells", cells)
    g.set_schedule("neighbor filter", 0 if form == "exact" else 1)
    g.build_neighbors()
    o.build_neighbors()
    assert o.num_pairs() > ns.n
    _same_connectivity(g, o)


def test_pairs_across_large_cells(gpu_lib, pkg):
    """A few nodes in a box of many reaches: the first build's cells are thousands
    of reaches wide, and pairs just within reach lie across a cell's face."""
    gen, abi = pkg.generators, pkg.abi
    pairs, h = 400, 1.0055e-6
    n = 2 * pairs + 2
    # the first build's cell edge (plan_capacities, setGrid)
    ghosts = n // 2 + 4096
    cells = (n + ghosts + ghosts // 2 + 1024) // 2 + 65
    cell = 2.0 * h * 1.001
    while int(1.0 / cell + 1.0) ** 3 > cells:
        cell *= 1.26
    rng = np.random.default_rng(5)
    first = rng.uniform(0.05, 0.95, (pairs, 3))
    first[:, 0] = cell * rng.integers(1, int(1.0 / cell), pairs) - rng.uniform(0.0, 3.0e-3, pairs) * 2.0 * h
    second = first + np.array([0.99995 * 2.0 * h, 0.0, 0.0])
    pos = np.concatenate([[[0.0, 0.0, 0.0], [1.0, 1.0, 1.0]], first, second])
    H = np.zeros((n, 6))
    H[:, [0, 3, 5]] = 1.0 / h
    ns = gen.NodeSet(pos, np.zeros((n, 3)), np.full(n, 1.0 / n), np.ones(n), np.ones(n), H, cell)
    g = pkg.SPHHydro(gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, periodic=(0, 0, 0)), ns)
    g.set_schedule("neighbor walk", 2)
    g.build_neighbors()
    off, nbr, _ = g.connectivity()
    # every node of a pair has the other one (none of the random pairs meet), the corners nobody
    near = np.sqrt(((pos[:, None] - pos[None]) ** 2).sum(2)) <= 2.0 * h
    np.fill_diagonal(near, False)
    assert near.sum() == 2 * pairs and not near[:2].any()
    assert np.array_equal(np.diff(off), near.sum(1)) and np.array_equal(nbr, np.nonzero(near)[1])


@pytest.mark.parametrize("passes", [1, 2])
def test_crowded_cells_appear(gpu_lib, pkg, oracle_mod, passes):
    """Crowded cells that no earlier build of the problem had (their block walks
    them), then the builds after it (their slots are listed), then none again."""
    ns, cfg = _clump(pkg, 300, 11, (1, 1, 1), True)
    rng = np.random.default_rng(3)
    spread = pkg.generators.NodeSet(rng.uniform(0.0, 1.0, (ns.n, 3)), ns.vel, ns.mass, ns.rho, ns.eps, ns.H, ns.dx)
    g = pkg.SPHHydro(cfg, spread)
    g.set_schedule("neighbor walk", 2)
    g.set_schedule("neighbor passes", passes)
    for nodes in (spread, ns, spread):
        g.set_state(nodes)
        o = oracle_mod.OracleProblem(cfg, nodes)
        o.build_neighbors()
        for _ in range(2):
            g.build_neighbors()
            _same_connectivity(g, o)


@pytest.mark.parametrize("nPerh", [2.0, 3.0])
def test_dense_sets(gpu_lib, pkg, oracle_mod, nPerh):
    """64 and 216 nodes per cell in the automatic schedule: the thread walk, the
    cell walk with every cell crowded, half-reach cells, then the steps' rebuilds,
    in a batch with a set that keeps the cell walk."""
    gen, abi = pkg.generators, pkg.abi
    ns = gen.kelvin_helmholtz(nx=15, ny=15, nz=15, nPerh=nPerh, jitter=0.1)
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, nPerh=nPerh, max_neighbors=2048, dtMin=1.0e-4, dtMax=1.0e-4)
    g = pkg.SPHHydro(cfg, ns)
    o = oracle_mod.OracleProblem(cfg, ns)
    o.build_neighbors()
    cells = []
    for _ in range(4):
        g.build_neighbors()
        _same_connectivity(g, o)
        cells.append(g.schedule("neighbor cells"))
    assert cells[0] == 1 and cells[-1] == 2
    box = ((0.0, 0.0, 0.0), (1.0, 0.25, 0.25))
    tube = gen.sod(nx=32, ny=8, nz=8, box=box)
    tcfg = gen.sod_config(abi, ns_box=box)
    pair = [pkg.SPHHydro(cfg, ns), pkg.SPHHydro(tcfg, tube)]
    alone = [g, pkg.SPHHydro(tcfg, tube)]
    g.set_state(ns)
    for h in alone:
        h.step(3)
    pkg.SPHBatch(pair).step(3)
    for a, b in zip(alone, pair):
        for k in ("position", "velocity", "mass density", "specific thermal energy", "H"):
            assert np.array_equal(a.field(k), b.field(k)), k


def test_autotune_of_a_dense_set(gpu_lib, pkg):
    """The autotuner compares the cells it says it compares: 216 nodes per cell walk
    faster over half-reach cells by half and more, also where the automatic
    schedule has taken them already."""
    gen, abi = pkg.generators, pkg.abi
    ns = gen.kelvin_helmholtz(nx=32, ny=32, nz=32, nPerh=3.0)
    g = pkg.SPHHydro(gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, nPerh=3.0, max_neighbors=2048), ns)
    for _ in range(3):
        g.build_neighbors()
    assert g.schedule("neighbor cells") == 2
    rep = g.autotune()
    assert rep["neighbor cells"] == 2 and rep["neighbor cells ms"][2] < 0.9 * rep["neighbor cells ms"][1]


def _windows(o, ns, reach, periodic):
    """Nodes of each cell, and for every cell with an internal node the nodes of its 27-cell window and those of
    them within reach of the cell (setGrid, nbr_cell_kernel)."""
    pos = np.concatenate([ns.pos, o.ghost_positions()])
    lo, hi = ns.pos.min(0), ns.pos.max(0)
    for a in range(3):
        if periodic[a]:
            lo[a], hi[a] = min(lo[a], -1.001 * reach), max(hi[a], 1.0 + 1.001 * reach)
    edge = 1.001 * reach
    dim = ((hi - lo) / edge).astype(int) + 1
    at = np.clip(((pos - lo) / edge).astype(int), 0, dim - 1)
    cells = {}
    for k, c in enumerate(map(tuple, at)):
        cells.setdefault(c, []).append(k)
    staged, tested = [], []
    for c in set(map(tuple, at[:ns.n])):
        window = [k for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)
                  for k in cells.get((c[0] + dx, c[1] + dy, c[2] + dz), [])]
        corner = lo + np.array(c) * edge
        gap = np.maximum(np.maximum(corner - pos[window], pos[window] - corner - edge), 0.0)
        staged.append(len(window))
        tested.append(int(((gap ** 2).sum(1) <= reach ** 2).sum()))
    return max(map(len, cells.values())), np.array(staged), np.array(tested)


# windows whose candidates need up to 32 ballot words; more candidates than ballot words hold; more nodes than the
# staging area holds: all with every cell in node order
@pytest.mark.parametrize("per_cell,branch", [(47.5, "words"), (54.0, "tested"), (63.0, "staged")])
@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("periodic", [(1, 1, 1), (1, 0, 0)])
def test_full_windows(gpu_lib, pkg, oracle_mod, per_cell, branch, passes, periodic):
    gen, abi = pkg.generators, pkg.abi
    n = 3000
    rng = np.random.default_rng(17)
    h = 0.5 * (per_cell / n) ** (1.0 / 3.0) / 1.001
    H = np.zeros((n, 6))
    H[:, [0, 3, 5]] = 1.0 / h
    ns = gen.NodeSet(rng.uniform(0.0, 1.0, (n, 3)), np.zeros((n, 3)), np.full(n, 1.0 / n), np.ones(n), np.ones(n), H, h)
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, periodic=periodic, max_neighbors=2048)
    o = oracle_mod.OracleProblem(cfg, ns)
    o.build_neighbors()
    largest, staged, tested = _windows(o, ns, 2.0 * h, periodic)
    assert largest <= 128
    if branch == "words":
        assert ((staged <= 1536) & (tested > 992) & (tested <= 1024)).any()
    elif branch == "tested":
        assert ((staged <= 1536) & (tested > 1024)).any() and (tested <= 1024).any()
    else:
        assert (staged > 1536).any() and (staged <= 1536).any()
    g = pkg.SPHHydro(cfg, ns)
    g.set_schedule("neighbor walk", 2)
    g.set_schedule("neighbor cells", 1)
    g.set_schedule("neighbor passes", passes)
    for _ in range(2):
        g.build_neighbors()
        _same_connectivity(g, o)


# (h 0.22: 85 nodes per cell, windows of 2,300)
@pytest.mark.parametrize("clump,h", [(300, 0.08), (0, 0.22)])
def test_crowded_cells_in_captured_steps(gpu_lib, pkg, clump, h):
    """Steps straight from a new state, whose first cell walk is in a captured step:
    a clump (the list joins the second capture) and a set that is crowded all over
    (half-reach cells from then on) take the states of eager steps."""
    gen, abi = pkg.generators, pkg.abi
    ns, _ = _clump(pkg, clump, 5, (1, 1, 1), False)
    ns.H[:, [0, 3, 5]] = 1.0 / h
    ns.pos[:] += np.random.default_rng(9).uniform(-1.0e-3, 1.0e-3, ns.pos.shape)
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, max_neighbors=2048, HUpdate=abi.H_INTEGRATE,
                        dtMin=1.0e-6, dtMax=1.0e-6)
    out = []
    for graph in (0, 1):
        g = pkg.SPHHydro(cfg, ns)
        g.set_schedule("neighbor walk", 0 if clump == 0 else 2)
        g.set_schedule("step graph", graph)
        g.step(9)
        out.append(g)
    assert out[0].schedule("neighbor cells") == out[1].schedule("neighbor cells") == (2 if clump == 0 else 1)
    assert np.array_equal(out[0].connectivity()[1], out[1].connectivity()[1])
    for k in ("position", "velocity", "mass density", "specific thermal energy", "H"):
        assert np.array_equal(out[0].field(k), out[1].field(k)), k
