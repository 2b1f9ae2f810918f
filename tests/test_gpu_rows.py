"""The group-of-lanes kernels (rows of 32 entries and more) at the edges of their
batches of 16 entries and their blocks of 8 nodes, and of 16 from 18,944 nodes
on.  The FP64 pair kernel forms the same terms and adds them in the same order
as the oracle, so every derivative is bit-equal except the cube root of the
ideal-H moment (CUDA pow against glibc pow, 2 ulp: 1e-12 is the specification's
tolerance)."""
import numpy as np
import pytest

from conftest import normwise

pytestmark = pytest.mark.gpu

KEYS = ["delta velocity hydro", "delta specific thermal energy", "delta mass density", "new mass density",
        "normalization", "velocity gradient", "M SPH gradient correction", "mass second moment",
        "max viscous pressure", "effective viscous pressure", "viscous work rate", "XSPH weight sum",
        "XSPH delta vi"]


# nodes: full blocks of 8, one node more than a full block (449, 497, 505)
@pytest.mark.parametrize("keep", [512, 505, 497, 449])
@pytest.mark.parametrize("options", [{}, {"XSPH": 1}, {"epsTensile": 0.3, "compatibleEnergyEvolution": 0},
                                     {"balsaraShearCorrection": 1}])
def test_rows(gpu_lib, pkg, oracle_mod, keep, options):
    gen, abi = pkg.generators, pkg.abi
    ns = gen.kelvin_helmholtz(nx=8, ny=8, nz=8, jitter=0.2, seed=keep)
    sel = np.sort(np.random.default_rng(keep).permutation(ns.n)[:keep])
    # rows of about 30 to 150 entries: smoothing scales spread by 1.7
    h = np.random.default_rng(keep + 1).uniform(0.13, 0.22, keep)
    H = np.zeros((keep, 6))
    H[:, [0, 3, 5]] = 1.0 / h[:, None]
    ns = gen.NodeSet(ns.pos[sel], ns.vel[sel], ns.mass[sel], ns.rho[sel], ns.eps[sel], H, ns.dx)
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, **options)
    g, o = pkg.SPHHydro(cfg, ns), oracle_mod.OracleProblem(cfg, ns)
    for p in (g, o):
        p.build_neighbors()
    off, _, _ = g.connectivity()
    rows = np.diff(off)
    assert rows.mean() >= 32 and len(set((rows % 16).tolist())) == 16      # every remainder of a batch
    if options.get("balsaraShearCorrection"):
        # the correction reads the last evaluation's velocity gradient
        g.initialize(), o.initialize()
    g.evaluateDerivatives()
    o.evaluate_derivatives()
    for k in KEYS:
        assert np.array_equal(g.field(k), o.field(k)), k
    assert normwise(g.field("new H"), o.field("new H")) <= 1e-12


@pytest.mark.parametrize("keep", [512, 505, 449])
@pytest.mark.parametrize("options", [{}, {"XSPH": 1, "compatibleEnergyEvolution": 0}, {"epsTensile": 0.3}])
def test_rows_mixed(gpu_lib, pkg, keep, options):
    """The mixed form's row kernel at the same edges: within the mixed form's
    1e-5 (normwise) of the FP64 form."""
    gen, abi = pkg.generators, pkg.abi
    ns = gen.kelvin_helmholtz(nx=8, ny=8, nz=8, jitter=0.2, seed=keep)
    ns = gen.NodeSet(ns.pos[:keep], ns.vel[:keep], ns.mass[:keep], ns.rho[:keep], ns.eps[:keep], ns.H[:keep], ns.dx)
    ns.H[:, [0, 3, 5]] = 1.0 / np.random.default_rng(keep).uniform(0.13, 0.22, keep)[:, None]
    out = {}
    for precision in (abi.PRECISION_FP64, abi.PRECISION_MIXED):
        g = pkg.SPHHydro(gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, precision=precision, **options), ns)
        g.build_neighbors()
        assert np.diff(g.connectivity()[0]).mean() >= 32
        g.evaluateDerivatives()
        out[precision] = {k: g.field(k) for k in KEYS + ["new H"]}
    for k, want in out[abi.PRECISION_FP64].items():
        assert normwise(out[abi.PRECISION_MIXED][k], want) <= 1e-5, k


@pytest.mark.parametrize("keep", [512, 505, 449])
def test_row_sums(gpu_lib, pkg, oracle_mod, keep):
    """Summed density, compatible energy and dt vote with 16 lanes per node over
    three RK2 steps: the oracle's states within the specification's 1e-12."""
    gen, abi = pkg.generators, pkg.abi
    ns = gen.kelvin_helmholtz(nx=8, ny=8, nz=8, jitter=0.1, seed=keep)
    ns = gen.NodeSet(ns.pos[:keep], ns.vel[:keep], ns.mass[:keep], ns.rho[:keep], ns.eps[:keep], ns.H[:keep], ns.dx)
    ns.H[:, [0, 3, 5]] = 1.0 / np.random.default_rng(keep).uniform(0.15, 0.2, keep)[:, None]
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, nPerh=1.51)
    g, o = pkg.SPHHydro(cfg, ns), oracle_mod.OracleProblem(cfg, ns)
    g.step(3)
    o.step(3)
    assert np.diff(g.connectivity()[0]).mean() >= 32
    for k in ("position", "velocity", "mass density", "specific thermal energy", "H"):
        assert normwise(g.field(k), o.field(k)) <= 1e-12, k
    assert abs(g.dt() - o.dt()) <= 1e-12 * o.dt()


@pytest.mark.parametrize("precision", ["PRECISION_FP64", "PRECISION_MIXED"])
def test_long_and_short_rows_in_one_batch(gpu_lib, pkg, precision):
    """A batch of a member with long rows and one with short rows: both equal
    their runs alone bit for bit."""
    gen, abi = pkg.generators, pkg.abi
    box = ((0.0, 0.0, 0.0), (1.0, 0.25, 0.25))

    def members():
        return [pkg.SPHHydro(gen.sod_config(abi, ns_box=box, precision=getattr(abi, precision)),
                             gen.sod(nx=32, ny=8, nz=8, box=box)),
                pkg.SPHHydro(gen.kh_config(abi, precision=getattr(abi, precision)),
                             gen.kelvin_helmholtz(nx=13, ny=13, nz=13, seed=3, jitter=0.1))]

    alone, together = members(), members()
    for h in alone:
        h.step(4)
    pkg.SPHBatch(together).step(4)
    for a, b in zip(alone, together):
        for k in ("position", "velocity", "mass density", "specific thermal energy", "H"):
            assert np.array_equal(a.field(k), b.field(k)), k


@pytest.mark.parametrize("precision", ["PRECISION_FP64", "PRECISION_MIXED"])
def test_paired_planes_of_large_problems(gpu_lib, pkg, precision):
    """The record layout of problems above 1.08M nodes: one step of the nodes of a
    cube far from the periodic planes equals the step of that cube alone, which
    keeps the small layout, bit for bit where the cube's surface (four kernel
    reaches) has no influence: neighbors, their order and every term are the same."""
    gen, abi = pkg.generators, pkg.abi
    cfg = gen.kh_config(abi, precision=getattr(abi, precision), dtMin=1.0e-4, dtMax=1.0e-4)
    whole = gen.kelvin_helmholtz(nx=104, ny=104, nz=104)
    assert 1.75 * whole.n > 1.9e6
    sel = np.flatnonzero((np.abs(whole.pos - 0.5) < 0.17).all(axis=1))
    cube = gen.NodeSet(whole.pos[sel], whole.vel[sel], whole.mass[sel], whole.rho[sel], whole.eps[sel],
                       whole.H[sel], whole.dx)
    # a reach is at most 2.7 spacings of 1/104
    inner = np.flatnonzero((np.abs(cube.pos - 0.5) < 0.17 - 4 * 2.7 / 104).all(axis=1))
    assert inner.size > 1000
    large, small = pkg.SPHHydro(cfg, whole), pkg.SPHHydro(cfg, cube)
    large.step(1)
    small.step(1)
    for k in ("position", "velocity", "mass density", "specific thermal energy", "H"):
        assert np.array_equal(large.field(k)[sel][inner], small.field(k)[inner]), k


@pytest.mark.parametrize("first,then", [(0.17, 0.1), (0.1, 0.17)])
def test_captured_step_follows_the_row_length(gpu_lib, pkg, first, then):
    """A new state in the same buffers with long rows in place of short ones, or
    the other way round: the steps after it run the kernels that a new problem
    of that state runs (the captured step of the old rows is right, but slow)."""
    gen, abi = pkg.generators, pkg.abi

    def state(h):
        ns = gen.kelvin_helmholtz(nx=8, ny=8, nz=8, jitter=0.1)
        ns.H[:, [0, 3, 5]] = 1.0 / h
        return ns

    # H follows the density, not the ideal neighbor count: the rows keep their length
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, HUpdate=abi.H_INTEGRATE, dtMin=1.0e-4, dtMax=1.0e-4)
    launches = []
    for states in ((first, then), (then,)):
        g = pkg.SPHHydro(cfg, state(max(first, then)))
        g.build_neighbors()                    # (both problems' buffers hold the long rows)
        for h in states:
            g.set_state(state(h))
            g.step(6)
            g.step(6)
        before = g.kernel_launches()
        g.step(6)
        launches.append(g.kernel_launches() - before)
        rows = np.diff(g.connectivity()[0]).mean()
        assert (rows >= 32) == (then > 0.15)
    assert launches[0] == launches[1]


@pytest.mark.parametrize("threads", [64, 128])
def test_autotune_leaves_the_pair_loop_of_long_rows(gpu_lib, pkg, threads):
    """The kernels with a group of lanes per node have no choice of threads: the
    autotuner reports one time and keeps the caller's value."""
    gen, abi = pkg.generators, pkg.abi
    box = ((0.0, 0.0, 0.0), (1.0, 0.25, 0.25))
    g = pkg.SPHHydro(gen.sod_config(abi, ns_box=box), gen.sod(nx=32, ny=8, nz=8, box=box))
    g.set_schedule("pair loop", threads)
    g.build_neighbors()
    rep = g.autotune()
    assert rep["pair loop"] == threads and g.schedule("pair loop") == threads
    assert rep["pair loop ms"][64] == rep["pair loop ms"][128] > 0


def _ragged(pkg, n, seed):
    """n nodes of a jittered 27^3 lattice in the unit cube, rows of about 40 entries."""
    gen = pkg.generators
    ns = gen.kelvin_helmholtz(nx=27, ny=27, nz=27, nPerh=1.1, jitter=0.1, seed=seed)
    sel = np.sort(np.random.default_rng(seed).permutation(ns.n)[:n])
    return gen.NodeSet(ns.pos[sel], ns.vel[sel], ns.mass[sel], ns.rho[sel], ns.eps[sel], ns.H[sel], ns.dx)


# from 18,944 nodes the blocks have two nodes per group of lanes, 16 in all: every kind of last block (its first pass
# full or not, its second empty, with one node, with seven, all but one)
@pytest.mark.parametrize("n,options", [(18944, {}), (19009, {"XSPH": 1}), (19015, {"XSPH": 1}), (19016, {}),
                                       (19017, {"epsTensile": 0.3, "compatibleEnergyEvolution": 0}),
                                       (19023, {"XSPH": 1, "balsaraShearCorrection": 1})])
def test_rows_of_large_problems(gpu_lib, pkg, oracle_mod, n, options):
    """FP64 bit for bit with the oracle; the mixed form within its 1e-5 of FP64."""
    gen, abi = pkg.generators, pkg.abi
    ns = _ragged(pkg, n, n)
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, nPerh=1.1, **options)
    g, o = pkg.SPHHydro(cfg, ns), oracle_mod.OracleProblem(cfg, ns)
    for p in (g, o):
        p.build_neighbors()
    assert np.diff(g.connectivity()[0]).mean() >= 32
    if options.get("balsaraShearCorrection"):
        g.initialize(), o.initialize()
    g.evaluateDerivatives()
    o.evaluate_derivatives()
    for k in KEYS:
        assert np.array_equal(g.field(k), o.field(k)), k
    assert normwise(g.field("new H"), o.field("new H")) <= 1e-12
    m = pkg.SPHHydro(gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, nPerh=1.1, precision=abi.PRECISION_MIXED, **options), ns)
    m.build_neighbors()
    if options.get("balsaraShearCorrection"):
        m.initialize()
    m.evaluateDerivatives()
    for k in KEYS + ["new H"]:
        assert normwise(m.field(k), g.field(k)) <= 1e-5, k


@pytest.mark.parametrize("n", [19009, 19015])
def test_ragged_steps_of_large_problems(gpu_lib, pkg, oracle_mod, n):
    """A step with the compatible energy of long rows at such sizes: the oracle's
    state within the specification's 1e-12."""
    gen, abi = pkg.generators, pkg.abi
    ns = _ragged(pkg, n, n)
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, nPerh=1.1)
    g, o = pkg.SPHHydro(cfg, ns), oracle_mod.OracleProblem(cfg, ns)
    g.step(1)
    o.step(1)
    for k in ("position", "velocity", "mass density", "specific thermal energy", "H"):
        assert normwise(g.field(k), o.field(k)) <= 1e-12, k


@pytest.mark.parametrize("precision", ["PRECISION_FP64", "PRECISION_MIXED"])
def test_uneven_batch_with_two_nodes_per_group(gpu_lib, pkg, precision):
    """Members of one node per group of lanes alone and of two in the batch (19,001
    nodes in all): bit for bit the same."""
    gen, abi = pkg.generators, pkg.abi
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, nPerh=1.1, XSPH=1, precision=getattr(abi, precision))

    def members():
        out = []
        for n in (7001, 6993, 5007):
            ns = _ragged(pkg, n, n)
            ns.H[:] *= (n / 19683.0) ** (1.0 / 3.0)          # (thinned: the rows keep their length)
            out.append(pkg.SPHHydro(cfg, ns))
        return out

    alone, together = members(), members()
    for h in alone:
        h.build_neighbors()
        assert np.diff(h.connectivity()[0]).mean() >= 32
        h.evaluateDerivatives()
    batch = pkg.SPHBatch(together)
    batch.build_neighbors()
    batch.evaluateDerivatives()
    for a, b in zip(alone, together):
        for k in KEYS + ["new H"]:
            assert np.array_equal(a.field(k), b.field(k)), k
    for h in alone:
        h.step(2)
    batch.step(2)
    for a, b in zip(alone, together):
        for k in ("position", "velocity", "mass density", "specific thermal energy", "H"):
            assert np.array_equal(a.field(k), b.field(k)), k


@pytest.mark.parametrize("precision", ["PRECISION_FP64", "PRECISION_MIXED"])
@pytest.mark.parametrize("options", [{}, {"XSPH": 1}, {"epsTensile": 0.3, "compatibleEnergyEvolution": 0},
                                     {"balsaraShearCorrection": 1}])
def test_rows_and_thread_kernels_give_the_same_bits(gpu_lib, pkg, precision, options):
    """The same rows with a group of lanes per node (a set alone: rows of 32 entries
    and more on average) and with a thread per node (the set with many isolated
    nodes behind it, which shorten the mean row): derivatives and steps are the same
    bits, summed density, compatible energy and update included."""
    gen, abi = pkg.generators, pkg.abi
    keep = 505
    ns = gen.kelvin_helmholtz(nx=8, ny=8, nz=8, jitter=0.2, seed=2)
    h = np.random.default_rng(4).uniform(0.13, 0.2, keep)
    H = np.zeros((keep, 6))
    H[:, [0, 3, 5]] = 1.0 / h[:, None]
    dense = gen.NodeSet(ns.pos[:keep], ns.vel[:keep], ns.mass[:keep], ns.rho[:keep], ns.eps[:keep], H, ns.dx)
    side = np.arange(22) + 2.0
    far = np.stack(np.meshgrid(side, side, side), -1).reshape(-1, 3)
    m = far.shape[0]

    def joined(a, fill):
        return np.concatenate([a, np.broadcast_to(fill, (m,) + a.shape[1:])])

    both = gen.NodeSet(np.concatenate([dense.pos, far]), joined(dense.vel, 0.0), joined(dense.mass, dense.mass[0]),
                       joined(dense.rho, 1.0), joined(dense.eps, 1.0), joined(dense.H, dense.H[0]), dense.dx)
    cfg = gen.kh_config(abi, kernel=abi.KERNEL_BSPLINE, periodic=(0, 0, 0), precision=getattr(abi, precision),
                        HUpdate=abi.H_INTEGRATE, dtMin=1.0e-4, dtMax=1.0e-4, **options)
    rows, threads = pkg.SPHHydro(cfg, dense), pkg.SPHHydro(cfg, both)
    for p, long in ((rows, True), (threads, False)):
        p.build_neighbors()
        entries = np.diff(p.connectivity()[0])
        assert (entries.mean() >= 32) == long and entries[:keep].mean() >= 32 and not entries[keep:].any()
        p.initialize()
        p.evaluateDerivatives()
    for k in KEYS + ["new H"]:
        assert np.array_equal(rows.field(k), threads.field(k)[:keep]), k
    for p in (rows, threads):
        p.step(3)
    for k in ("position", "velocity", "mass density", "specific thermal energy", "H"):
        assert np.array_equal(rows.field(k), threads.field(k)[:keep]), k
