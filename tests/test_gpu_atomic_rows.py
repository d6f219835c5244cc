"""The atomic executor's reductions on the GPU: rows of every width laid out
across warps of every fill, runs of neighbouring cells with one target point
summed before the reduction, and the contracted miniAero flux over states the
generator does not reach.  Tolerances as for every atomic run: 1e-12 (FP64)
and 1e-5 (FP32) normwise against the oracle's serial loop."""
import numpy as np
import pytest

from cuda_fot_b200 import meshgen as mg
from oracle import oracle_py as O
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


def F():
    from cuda_fot_b200 import fot
    return fot


def cut(md, n):
    """The mesh's first n cells (all points stay)."""
    md.n_cells = n
    md.maps = [np.ascontiguousarray(m[:n]) for m in md.maps]
    md.cell_data = [np.ascontiguousarray(d[:, :n]) for d in md.cell_data]
    return md


MESHES = {"res_calc": lambda lay: mg.res_calc(24, 20, 5, lay), "mini_aero": lambda lay: mg.mini_aero(8, 5, lay),
          "lulesh": lambda lay: mg.lulesh(9, 5, lay), "volna": lambda lay: mg.volna(20, 16, 5, lay),
          "getacc": lambda lay: mg.getacc(30, 22, 5, lay)}


def check(md, flags, iters=2):
    p = F().Problem.from_mesh(md)
    plan = p.plan(F().EXEC_ATOMIC, 256, flags)
    plan.run(iters)
    p.sync()
    assert rel_err(p.point_weights(0), O.serial(md, iters)[0][0]) <= (1e-5 if md.loop == mg.VOLNA else 1e-12)


@pytest.mark.parametrize("flags", [0, 1])
@pytest.mark.parametrize("layout", ["aos", "soa"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 600])
@pytest.mark.parametrize("name", list(MESHES))
def test_rows_of_partly_filled_warps(name, n, layout, flags):
    check(cut(MESHES[name](layout), n), flags)


# lengths of the runs of one target point that cells come in
RUNS = {"all_one": [10 ** 6], "pairs": [2], "threes": [3], "warp": [32], "across_warps": [33],
        "mixed": [1, 2, 1, 5, 3, 17, 1, 1, 8, 31, 4]}


@pytest.mark.parametrize("layout", ["aos", "soa"])
@pytest.mark.parametrize("runs", list(RUNS))
@pytest.mark.parametrize("name", ["volna", "getacc"])
def test_runs_of_one_point(name, runs, layout):
    md = MESHES[name](layout)
    g = np.random.default_rng(7)
    n, dim, points = md.n_cells, md.maps[0].shape[1], md.n_points[0]
    length = np.resize(np.array(RUNS[runs]), n)
    run = np.repeat(np.arange(n), length)[:n]
    # distinct points in a row; neighbouring runs may share a point by chance
    rows = np.stack([g.permutation(points)[:dim] for _ in range(int(run.max()) + 1)])
    m = np.ascontiguousarray(rows[run].astype(np.uint32))
    md.maps = [m] + [m.copy() for _ in md.maps[1:]]
    check(md, 0)


@pytest.mark.parametrize("layout", ["aos", "soa"])
def test_contracted_face_flux(layout):
    """Faces of any area and direction, slow to supersonic flow in each
    direction (every branch of the eigenvalue fix), steep gradients."""
    md = mg.mini_aero(9, 6, "aos")
    g = np.random.default_rng(11)
    rec, face = md.point_data[1], md.cell_data[0]
    n = len(rec)
    rho = g.uniform(0.2, 3.0, n)
    vel = g.uniform(-2.5, 2.5, (n, 3)) * g.choice([0.01, 0.3, 1.0, 4.0], (n, 1))
    rec[:, 0] = rho
    rec[:, 1:4] = rho[:, None] * vel
    rec[:, 4] = rho * (g.uniform(1.5, 4.0, n) + 0.5 * (vel ** 2).sum(1))
    rec[:, 8:20] = g.uniform(-2e-2, 2e-2, (n, 12))
    rec[:, 20:23] = g.uniform(-1e-3, 1e-3, (n, 3))  # of T, which is 2e-3 to 6e-3 here
    frame = np.linalg.qr(g.normal(size=(md.n_cells, 3, 3)))[0] * g.uniform(0.05, 5.0, (md.n_cells, 1, 3))
    face[3:12] = frame.transpose(2, 1, 0).reshape(9, -1)
    check(md.to_layout(layout), 1)


# meshes around the sizes at which the launch is split into phases: fewer
# tiles than the GPU holds CTAs, a few rounds, and more rounds than one phase
SIZES = {"getacc_small": lambda lay: mg.getacc(33, 21, 5, lay), "getacc_phases": lambda lay: mg.getacc(1100, 905, 5, lay),
         "volna_phases": lambda lay: mg.volna(1003, 997, 5, lay), "res_calc": lambda lay: mg.res_calc(301, 299, 5, lay),
         "res_calc_phases": lambda lay: mg.res_calc(811, 803, 5, lay),
         "mini_aero_phases": lambda lay: mg.mini_aero(103, 5, lay, permute=False),
         "lulesh": lambda lay: mg.lulesh(31, 5, lay)}


@pytest.mark.parametrize("iters", [1, 2, 5])
@pytest.mark.parametrize("layout", ["aos", "soa"])
@pytest.mark.parametrize("name", list(SIZES))
def test_iterations_of_one_launch(name, layout, iters):
    """Every cell once per iteration, in either direction through the mesh."""
    md = SIZES[name](layout)
    p = F().Problem.from_mesh(md)
    plan = p.plan(F().EXEC_ATOMIC, 256, F().PLAN_NO_AGGREGATE)
    plan.run(iters)
    p.sync()
    # rel_err is normwise, so one serial iteration scaled up serves as the
    # oracle of several: the loops never read what they increment (FP64: the
    # scaling rounds once; FP32 starts from a state of its own)
    base, one = md.point_data[0].astype(np.float64), O.serial(md, 1)[0][0].astype(np.float64)
    want = base + iters * (one - base)
    assert rel_err(p.point_weights(0), want) <= (1e-5 if md.loop == mg.VOLNA else 1e-12)


@pytest.mark.parametrize("layout", ["aos", "soa"])
@pytest.mark.parametrize("sizes", [(9, 14, 3), (420, 300, 3)])  # tiles of 256 and of 1,024 cells
def test_batch_tiles_of_either_size(sizes, layout):
    side, side2, pairs = sizes
    mds = [md for i in range(pairs)
           for md in (mg.res_calc(side, side - i, 5 + i, layout), mg.volna(side2, side2 + i, 5 + i, layout))]
    probs = [F().Problem.from_mesh(md) for md in mds]
    b = F().Batch([p.plan(F().EXEC_ATOMIC, 256) for p in probs])
    b.run(3)
    b.sync()
    for md, p in zip(mds, probs):
        assert rel_err(p.point_weights(0), O.serial(md, 3)[0][0]) <= (1e-5 if md.loop == mg.VOLNA else 1e-12)


@pytest.mark.parametrize("flags", [0, 1])
@pytest.mark.parametrize("runs", list(RUNS))
def test_quads_of_rows(runs, flags):
    """Rows of 4 doubles through the quads of a loop that gathers (res_calc, AOS)."""
    md = MESHES["res_calc"]("aos")
    g = np.random.default_rng(9)
    n, points = md.n_cells, md.n_points[0]
    run = np.repeat(np.arange(n), np.resize(np.array(RUNS[runs]), n))[:n]
    rows = np.stack([g.permutation(points)[:2] for _ in range(int(run.max()) + 1)])
    m = np.ascontiguousarray(rows[run].astype(np.uint32))
    md.maps = [m, md.maps[1], m.copy(), m.copy()]
    check(md, flags)
