"""Plans of meshes whose cells lie in no useful order run kernels of their own
(other registers per thread): the results are those of every other plan."""
import numpy as np
import pytest

from cuda_fot_b200 import meshgen as mg
from oracle import oracle_py as O
from tests.helpers import bitwise_equal, rel_err

pytestmark = pytest.mark.gpu


def F():
    from cuda_fot_b200 import fot
    return fot


def shuffled(md, seed=3):
    """The mesh's cells in random order."""
    order = np.random.default_rng(seed).permutation(md.n_cells)
    md.maps = [np.ascontiguousarray(m[order]) for m in md.maps]
    md.cell_data = [np.ascontiguousarray(d[:, order]) for d in md.cell_data]
    return md


@pytest.mark.parametrize("iters", [1, 3])
@pytest.mark.parametrize("layout", ["aos", "soa"])
@pytest.mark.parametrize("block", [64, 128, 256, 512])
@pytest.mark.parametrize("scattered", [False, True])
def test_coloured_blocks(scattered, block, layout, iters):
    md = mg.lulesh(17, 5, layout, permute=False)
    if scattered:
        md = shuffled(md)
    p = F().Problem.from_mesh(md)
    plan = p.plan(F().EXEC_HIER, block)
    st, ex = plan.stats(), plan.export()
    assert (st["avg_block_points"] * st["n_blocks"] > 4 * md.n_cells) == scattered
    plan.run(iters)
    p.sync()
    rep, rep_cd = O.replay_hier(md, ex, iters)
    assert bitwise_equal(p.point_weights(0), rep[0])
    got = np.empty_like(rep_cd[1])
    got[:, ex["cell_id"]] = p.cell_weights(1)
    assert bitwise_equal(got, rep_cd[1])


def sectors_per_warp(m, per_sector=4, warps=256):
    """Mean sectors that a slot's points of 32 neighbouring cells fall into,
    over groups of cells spread evenly over the mesh."""
    n = len(m)
    c = np.minimum(((n + 31) // 32 * np.arange(warps, dtype=np.int64) // warps * 32)[:, None] + np.arange(32), n - 1)
    return np.mean([len(np.unique(m[g, s] // per_sector)) for g in c for s in range(m.shape[1])])


@pytest.mark.parametrize("flags", [0, 1])
@pytest.mark.parametrize("n", [1, 32, 33, 64, 300, 1537, None])
@pytest.mark.parametrize("mesh", ["numbered_at_random", "cells_shuffled", "ordered"])
def test_atomic_rows(mesh, n, flags):
    import torch
    md = mg.mini_aero(14, 5, "soa", permute=mesh == "numbered_at_random")
    if mesh == "cells_shuffled":
        md = shuffled(md)
    if n is not None:
        md.n_cells = n
        md.maps = [np.ascontiguousarray(m[:n]) for m in md.maps]
        md.cell_data = [np.ascontiguousarray(d[:, :n]) for d in md.cell_data]
    p = F().Problem.from_mesh(md)
    plan = p.plan(F().EXEC_ATOMIC, 256, flags)
    # resident CTAs an SM of the two forms
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert plan.stats()["grid"] == (2 if sectors_per_warp(md.maps[0]) > 16 else 3) * sms
    if n is None:
        assert (plan.stats()["grid"] == 3 * sms) == (mesh == "ordered")
    plan.run(2)
    p.sync()
    assert rel_err(p.point_weights(0), O.serial(md, 2)[0][0]) <= 1e-12
    # the plan outlives a reordering, with the form that it was built with
    p.reorder(F().ORDER_RCM)
    plan.run(1)
    p.sync()
    got = p.point_weights(0)[:, p.point_permutation(0)]
    assert rel_err(got, O.serial(md, 3)[0][0]) <= 1e-12
