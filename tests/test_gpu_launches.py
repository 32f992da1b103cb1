"""kernel_launches of pgxc_timings: the kernels that a build launches, counted by the profiler."""
import numpy as np
import pytest

import oracle as O
from pgxc import cases, lib

pytestmark = pytest.mark.gpu


def _count(call):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA], acc_events=True) as prof:
        tm = call()
    kernels = [e for e in prof.events() if "CUDA" in str(e.device_type) and not e.name.startswith(("Mem", "Activity"))]
    if not kernels:
        pytest.skip("the profiler records no kernels here")
    return tm["kernel_launches"], len(kernels)


KINDS = [("VWN", 1), ("PBE", 1), ("PBE", 2), ("TPSS", 1), ("TPSS", 2)]
LAYOUTS = [("fp64", 0.0, False), ("fp64", 0.0, True), ("mixed", 1e-10, False), ("mixed", 1e-10, True)]
DENSE = [("fp64", -1.0, False), ("mixed", -1.0, False)]  # closed shell, no meta-GGAs


@pytest.mark.parametrize("chunk", [0, 1024])
@pytest.mark.parametrize("nocc", [3, 40], ids=["orbitals", "P"])
@pytest.mark.parametrize("functional,ispin,precision,threshold,keep",
                         [(*k, *layout) for k in KINDS for layout in LAYOUTS] +
                         [(*k, *layout) for k in KINDS[:2] for layout in DENSE])
def test_launches_are_counted(functional, ispin, precision, threshold, keep, nocc, chunk):
    c = cases.small_case(functional, seed=44, natoms=5, nocc=3, ispin=ispin)
    O.weight_case(c)
    c.nocc = nocc
    c.C = np.random.default_rng(2).normal(size=(c.nbas, nocc, ispin)) / c.nbas
    c.occ = np.ones((nocc, ispin))
    with lib.Context(c, precision=precision, screen_threshold=threshold, keep_orbitals=keep,
                     max_chunk_points=chunk) as ctx:
        ctx.build()
        told, launched = _count(lambda: ctx.build(timings=True)[3])
    assert told == launched
