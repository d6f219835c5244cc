"""The most iterations of one batched call: 2^32 tiles of 1,024 cells, whatever
tiles the batch runs by.  The accepted calls are captured and never replayed
(they would run for minutes); a refused one launches nothing."""
import pytest

from cuda_fot_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def test_small_tiles_do_not_lower_the_limit():
    import torch

    from cuda_fot_b200 import fot as F
    p = F.Problem.from_mesh(mg.res_calc(24, 20, 5))  # 916 edges: one tile of 1,024, four of 256
    b = F.Batch([p.plan(F.EXEC_ATOMIC, 256)])
    st = torch.cuda.Stream()
    b.run(1, st)
    torch.cuda.synchronize()
    for iterations in (2 ** 30 + 1, 2 ** 32 - 2 ** 20):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            b.run(iterations, st)
        del g
    with pytest.raises(F.FotError):
        b.run(2 ** 32 - 1, st)
    torch.cuda.synchronize()
