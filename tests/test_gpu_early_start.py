"""Calls behind a kernel that lets its dependents start at once and only then,
about 200 us later, writes what they read (an application's kernel built for
programmatic dependent launch does that): no launch of a call, the first or a
later one, may read before that kernel is complete."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from cuda_fot_b200 import meshgen as mg
from oracle import oracle_py as O
from tests.helpers import bitwise_equal, rel_err

pytestmark = pytest.mark.gpu

# one CTA; the delay is bounded by time and by a number of polls
SOURCE = r"""
#include <cuda_runtime.h>
__global__ void late_scale(double *v, unsigned n, double f, unsigned long long ns) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  unsigned long long t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (unsigned i = 0; i < (1u << 20); ++i) {
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t - t0 > ns) break;
  }
  for (unsigned i = threadIdx.x; i < n; i += blockDim.x) v[i] *= f;
}
extern "C" int launch_late_scale(double *v, unsigned n, double f, unsigned long long ns, cudaStream_t st) {
  late_scale<<<1, 512, 0, st>>>(v, n, f, ns);
  return (int)cudaGetLastError();
}
"""


def F():
    from cuda_fot_b200 import fot
    return fot


@pytest.fixture(scope="module")
def late_scale(tmp_path_factory):
    d = tmp_path_factory.mktemp("late_scale")
    (d / "late_scale.cu").write_text(SOURCE)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-shared",
                    "-Xcompiler", "-fPIC", "-o", str(d / "late_scale.so"), str(d / "late_scale.cu")], check=True)
    f = C.CDLL(str(d / "late_scale.so")).launch_late_scale
    f.argtypes = [C.c_void_p, C.c_uint, C.c_double, C.c_ulonglong, C.c_void_p]

    def launch(p, k, factor, st):
        n = int(np.prod(p.point_shape(k)))
        assert f(p.point_data_device(k), n, factor, 200_000, st.cuda_stream) == 0

    return launch


# mesh and the read dataset that is scaled (mini_aero's records and the
# nodes of LULESH scale as a whole; res_calc: its states q)
CASES = {"res_calc": (lambda lay: mg.res_calc(24, 20, 5, lay), 2), "mini_aero": (lambda lay: mg.mini_aero(8, 5, lay), 1),
         "lulesh": (lambda lay: mg.lulesh(8, 5, lay), 1)}


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("iters", [1, 2, 5])
@pytest.mark.parametrize("layout", ["aos", "soa"])
@pytest.mark.parametrize("plan", ["atomic", "coloured"])
@pytest.mark.parametrize("name", list(CASES))
def test_run_waits_for_what_precedes_it(late_scale, name, plan, layout, iters, captured):
    import torch
    make, k = CASES[name]
    md = make(layout)
    p = F().Problem.from_mesh(md)
    pl = p.plan(F().EXEC_HIER, 128) if plan == "coloured" else p.plan(F().EXEC_ATOMIC, 256)
    st = torch.cuda.Stream()
    # kernels are loaded on their first launch: not during the delay
    pl.run(iters, st)
    late_scale(p, k, 1.0, st)
    torch.cuda.synchronize()
    p.set_point_data(0, md.point_data[0])
    torch.cuda.synchronize()

    def calls():
        late_scale(p, k, 1.0625, st)
        pl.run(iters, st)

    if captured:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            calls()
        g.replay()
    else:
        calls()
    torch.cuda.synchronize()
    p.sync()
    if captured:
        del g
    md.point_data[k] = md.point_data[k] * 1.0625
    if plan == "coloured":
        assert bitwise_equal(p.point_weights(0), O.replay_hier(md, pl.export(), iters)[0][0])
    else:
        assert rel_err(p.point_weights(0), O.serial(md, iters)[0][0]) <= 1e-12


@pytest.mark.parametrize("plan", ["atomic", "coloured"])
def test_airfoil_waits_for_what_precedes_it(late_scale, plan):
    import torch
    md = mg.res_calc(24, 20, 5)
    extras = mg.airfoil_extras(md)
    p = F().Problem.from_mesh(md)
    pl = p.plan(F().EXEC_HIER, 128) if plan == "coloured" else p.plan(F().EXEC_ATOMIC, 256)
    a = F().Airfoil(p, **extras)
    st = torch.cuda.Stream()
    a.run(pl, 2, st, rms=False)
    late_scale(p, 2, 1.0, st)
    torch.cuda.synchronize()
    for k in (0, 2):
        p.set_point_data(k, md.point_data[k])
    torch.cuda.synchronize()
    late_scale(p, 2, 1.0625, st)
    a.run(pl, 2, st, rms=False)
    torch.cuda.synchronize()
    p.sync()
    md.point_data[2] = md.point_data[2] * 1.0625
    if plan == "coloured":
        assert bitwise_equal(p.point_weights(2), O.airfoil(md, extras, 2, pl.export())[0][2])
    else:
        assert rel_err(p.point_weights(2), O.airfoil(md, extras, 2)[0][2]) <= 1e-11


@pytest.mark.parametrize("plan", ["atomic", "coloured"])
def test_batch_waits_for_what_precedes_it(late_scale, plan):
    import torch
    mds = [mg.res_calc(24, 20, 5), mg.res_calc(17, 9, 6)]
    probs = [F().Problem.from_mesh(md) for md in mds]
    plans = [p.plan(F().EXEC_HIER, 128) if plan == "coloured" else p.plan(F().EXEC_ATOMIC, 256) for p in probs]
    b = F().Batch(plans)
    st = torch.cuda.Stream()
    b.run(3, st)
    late_scale(probs[0], 2, 1.0, st)
    torch.cuda.synchronize()
    for md, p in zip(mds, probs):
        p.set_point_data(0, md.point_data[0])
    torch.cuda.synchronize()
    for p in probs:
        late_scale(p, 2, 1.0625, st)
    b.run(3, st)
    b.sync(st)
    for md, p, pl in zip(mds, probs, plans):
        md.point_data[2] = md.point_data[2] * 1.0625
        if plan == "coloured":
            assert bitwise_equal(p.point_weights(0), O.replay_hier(md, pl.export(), 3)[0][0])
        else:
            assert rel_err(p.point_weights(0), O.serial(md, 3)[0][0]) <= 1e-12
