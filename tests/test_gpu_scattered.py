"""Plans of meshes whose cells lie in no useful order run kernels of their own
(other registers per thread): the results are those of every other plan."""
import numpy as np
import pytest

from cuda_fot_b200 import meshgen as mg
from oracle import oracle_py as O
from tests.helpers import bitwise_equal

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
