"""Engine calls captured by the caller, after work of other kinds on the
stream: their kernels start while the one before them drains, which must hold
as well after a copy, a memset, a join of two streams and nothing at all, and
after a kernel that writes what they read."""
import numpy as np
import pytest

from cuda_fot_b200 import meshgen as mg
from tests.helpers import bitwise_equal, rel_err

pytestmark = pytest.mark.gpu


def F():
    from cuda_fot_b200 import fot
    return fot


class View:
    def __init__(self, p, k):
        self.__cuda_array_interface__ = {"shape": p.point_shape(k), "typestr": np.dtype(p.point_dtype(k)).str,
                                         "data": (p.point_data_device(k), False), "version": 3}


def view(p, k):
    import torch
    return torch.as_tensor(View(p, k), device="cuda")


PLANS = {"atomic": (0, 0), "coloured": (1, 0)}


@pytest.mark.parametrize("before", ["nothing", "memset", "copy", "kernel", "join"])
@pytest.mark.parametrize("plan", list(PLANS))
def test_capture_after(plan, before):
    import torch
    md = mg.res_calc(61, 47, 5)
    results = []
    for captured in (False, True):
        p = F().Problem.from_mesh(md)
        pl = p.plan(PLANS[plan][0], 128 if PLANS[plan][0] else 256, PLANS[plan][1])
        res, q = view(p, 0), view(p, 2)
        fresh = q.clone() * 1.25
        other = torch.cuda.Stream()
        work = torch.cuda.Stream()

        def calls(st):
            if before == "memset":
                res.zero_()
            elif before == "copy":
                q.copy_(fresh, non_blocking=True)
            elif before == "kernel":
                q.mul_(1.25)
            elif before == "join":
                other.wait_stream(st)
                with torch.cuda.stream(other):
                    q.mul_(1.25)
                res.add_(1.0)
                st.wait_stream(other)
            pl.run(2, st)

        torch.cuda.synchronize()
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=work):
                calls(work)
            g.replay()
        else:
            work.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(work):
                calls(work)
        torch.cuda.synchronize()
        results.append(p.point_weights(0))
        if captured:
            del g
    if plan == "coloured":
        assert bitwise_equal(*results)
    else:
        assert rel_err(*results) <= 1e-12


def test_airfoil_and_batch_after_a_copy():
    import torch
    md = mg.res_calc(61, 47, 5)
    ex = mg.airfoil_extras(md)
    out = []
    for captured in (False, True):
        p = F().Problem.from_mesh(md)
        pl = p.plan(F().EXEC_HIER, 128)
        a = F().Airfoil(p, **ex)
        b = F().Problem.from_mesh(mg.volna(31, 30, 5))
        batch = F().Batch([b.plan(F().EXEC_ATOMIC, 256)])
        q, fresh = view(p, 2), view(p, 2).clone() * 1.01
        st = torch.cuda.Stream()

        def calls():
            q.copy_(fresh, non_blocking=True)
            a.run(pl, 2, st, rms=False)
            view(b, 0).add_(0.5)
            batch.run(2, st)

        torch.cuda.synchronize()
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                calls()
            g.replay()
        else:
            with torch.cuda.stream(st):
                calls()
        torch.cuda.synchronize()
        out.append((p.point_weights(2), b.point_weights(0)))
        if captured:
            del g
    assert bitwise_equal(out[0][0], out[1][0])
    assert rel_err(out[0][1], out[1][1]) <= 1e-5
