"""An object is ready for any stream when its creation returns, also while the
default stream, on which its buffers are filled, has work of its own: a run on
a non-blocking stream does not wait for that stream."""
import threading

import pytest

from cuda_fot_b200 import meshgen as mg
from oracle import oracle_py as O
from tests.helpers import bitwise_equal, rel_err

pytestmark = pytest.mark.gpu


def F():
    from cuda_fot_b200 import fot
    return fot


class BusyDefaultStream:
    """Keeps a few kernels of about a millisecond queued on the default stream
    from another thread."""

    def __enter__(self):
        import torch
        self.stop, started = threading.Event(), threading.Event()

        def work():
            queued = []
            while not self.stop.is_set():
                torch.cuda._sleep(2_000_000)
                queued.append(torch.cuda.Event())
                queued[-1].record()
                started.set()
                if len(queued) > 4:
                    queued.pop(0).synchronize()

        self.thread = threading.Thread(target=work)
        self.thread.start()
        started.wait()

    def __exit__(self, *_):
        self.stop.set()
        self.thread.join()


def test_airfoil_rms_counts_from_zero():
    import torch
    md = mg.res_calc(40, 32, 6)
    ex = mg.airfoil_extras(md)
    p = F().Problem.from_mesh(md)
    plan = p.plan(F().EXEC_HIER, 128)
    st = torch.cuda.Stream()
    with BusyDefaultStream():
        af = F().Airfoil(p, **ex)
        af.run(plan, 2, st, rms=False)
        st.synchronize()
    torch.cuda.synchronize()
    ref, rms = O.airfoil(md, ex, 2, plan.export())
    assert bitwise_equal(p.point_weights(2), ref[2])
    assert abs(af.rms() - rms) <= 1e-12 * rms
    af.run(plan, 1, st, rms=False)
    ref, rms = O.airfoil(md, ex, 3, plan.export())
    assert abs(af.rms(st) - rms) <= 1e-12 * rms


@pytest.mark.parametrize("kernel", ["atomic", "coloured"])
def test_batch_starts_from_a_clear_queue(kernel):
    import torch
    mds = [mg.res_calc(24, 20, 5), mg.res_calc(17, 9, 6)]
    probs = [F().Problem.from_mesh(md) for md in mds]
    plans = [p.plan(F().EXEC_HIER, 128) if kernel == "coloured" else p.plan(F().EXEC_ATOMIC, 256) for p in probs]
    st = torch.cuda.Stream()
    with BusyDefaultStream():
        b = F().Batch(plans)
        b.run(2, st)
        st.synchronize()
    torch.cuda.synchronize()
    b.run(1, st)
    b.sync(st)
    for md, p, plan in zip(mds, probs, plans):
        if kernel == "coloured":
            assert bitwise_equal(p.point_weights(0), O.replay_hier(md, plan.export(), 3)[0][0])
        else:
            assert rel_err(p.point_weights(0), O.serial(md, 3)[0][0]) <= 1e-12
