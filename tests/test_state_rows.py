"""State transfer by rows (k_state_rows): any subset of fields of any scene, in creation order, after a re-binning has
permuted the particles."""
import ctypes as C

import numpy as np
import pytest

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200 import scenes as S
from mpm_cuda_b200.sim import Scene, Simulation

from helpers import group_from_arrays


def scene(d, n, seed):
    rng = np.random.default_rng(seed)
    h = 1.0 / 32
    x = 0.3 + 0.4 * rng.random((n, d))
    F = np.eye(d) + 0.02 * rng.standard_normal((n, d, d))
    g = group_from_arrays(S.jello(), h, 8, x, rng.standard_normal((n, d)), rng.standard_normal((n, d, d)), F, np.ones(n))
    g.aux = None
    return Scene(dim=d, n=(32,) * d, h=h, dt=1e-5, groups=[g])


@pytest.mark.gpu
@pytest.mark.parametrize("d", [3, 2])
@pytest.mark.parametrize("n", [2, 31, 257])
def test_subsets_of_fields_of_one_scene(gpu, d, n):
    scs = [scene(d, 65, 1), scene(d, n, 2), scene(d, 40, 3)]
    widths = {"x": d, "v": d, "C": d * d, "F": d * d, "aux": 1}
    with Simulation(scs, kernel_config=24) as sim:
        sim.step(3)
        before = [sim.get_state(k) for k in range(3)]
        for name in widths:  # one field at a time gives what all at once gave
            out = np.full((n, widths[name]), np.nan, np.float32)
            ptr = [L.fptr(out) if name == f else None for f in widths]
            assert sim._lib.mpm_get_state(sim.handle, 1, *ptr) == L.OK
            np.testing.assert_array_equal(out.ravel(), before[1][name].ravel())
        rng = np.random.default_rng(4)
        new = {"v": np.float32(rng.standard_normal((n, d))), "F": np.float32(rng.standard_normal((n, d, d)))}
        sim.set_state(1, v=new["v"], F=new["F"])
        after = [sim.get_state(k) for k in range(3)]
        for k in range(3):
            for name in widths:
                want = new[name] if k == 1 and name in new else before[k][name]
                np.testing.assert_array_equal(after[k][name], want)
