"""Calls on a live handle queue their device work on the handle's stream, which does not wait for the default stream."""
import os
import re

import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import group_from_arrays

ENGINE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpm_cuda_b200", "csrc",
                      "mpm_engine.cu")


def engine_functions():
    """{name: body} of the engine's member functions."""
    with open(ENGINE) as f:
        parts = re.split(r"\n(?=(?:int|void|bool|FusedArgs) Engine::\w+\()", f.read())
    return {re.match(r"\w+ Engine::(\w+)\(", p).group(1): p for p in parts[1:]}


def test_no_write_on_the_default_stream():
    """Only mpm_create, which waits for the device before it returns, may clear or fill device memory on the default
    stream: such a call returns before the work is done, and the handle's stream does not wait for it.  (A copy to the
    host returns when the data is there.)"""
    functions = engine_functions()
    assert len(functions) > 30 and "alloc_det" in functions
    for name, body in functions.items():
        if name == "create":
            continue
        code = re.sub(r"//[^\n]*", "", body)
        assert not re.search(r"\bcudaMemset\(", code), name
        for call in re.findall(r"\bcudaMemcpy\([^;]*;", code):
            assert "cudaMemcpyDeviceToHost" in call, (name, call)
        for launch in re.findall(r"<<<([^;]*?)>>>", code, re.S):
            assert re.search(r",\s*(stream|copy_stream)\s*$", launch), (name, launch)


@pytest.mark.gpu
@pytest.mark.parametrize("d,n_grid", [(3, 64), (2, 256)])
def test_deterministic_mode_of_a_live_handle(gpu, d, n_grid):
    """A handle that turns deterministic while the caller's own work occupies the default stream gives the bits of one
    that was created so: before its first substep, and after substeps that permuted the particles."""
    import torch
    h = 1.0 / n_grid
    x, v, C, F, aux = S.perturbed_blob(d, S.jello(), n_grid=n_grid, h=h, ppc=8, radius_cells=9.0, seed=5,
                                       center=np.full(d, 0.5))
    sc = Scene(dim=d, n=(n_grid,) * d, h=h, dt=5e-5, groups=[group_from_arrays(S.jello(), h, 8, x, v, C, F, aux)],
               bc_type=L.BC_SLIP, bc_lo=3, bc_hi=3)
    for before in (0, 3):
        with Simulation([sc], kernel_config=25) as sim, Simulation([sc], p2g_mode=L.P2G_DETERMINISTIC) as ref:
            if before:
                sim.step(before)
                s = sim.get_state(0)
                ref.set_state(0, x=s["x"], v=s["v"], C_=s["C"], F=s["F"], aux=s["aux"])
            torch.cuda._sleep(200_000_000)  # about a tenth of a second on the default stream
            sim.set_p2g_mode(L.P2G_DETERMINISTIC)
            sim.step(4)
            torch.cuda.synchronize()
            ref.step(4)
            assert sim.device_errors() == 0 and ref.device_errors() == 0
            got, want = sim.get_state(0), ref.get_state(0)
            for q in ("x", "v", "C", "F", "aux"):
                assert np.array_equal(got[q], want[q]), (before, q)
