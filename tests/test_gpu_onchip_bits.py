"""The on-chip kernel gives the bits of a launch per step: reference mode, whose
arithmetic is left to the compiler's contraction, all collision models; and the
largest lattices that fit, and the first that do not."""
import numpy as np
import pytest

from thesis_gb300 import lattice
from thesis_gb300 import native as N
from thesis_gb300.solver import Arguments, Solver

pytestmark = pytest.mark.gpu


def state(monkeypatch, kernel, lat, args, steps):
    if kernel:
        monkeypatch.setenv("THESIS_LBM_KERNEL", kernel)
    else:
        monkeypatch.delenv("THESIS_LBM_KERNEL", raising=False)
    nn = lat.num_nodes
    rng = np.random.default_rng(5)
    u = np.where(lat.node_type == 1, 0.02 * rng.standard_normal(nn), 0.0)
    with Solver(lat, args) as s:
        on_chip = s.on_chip
        s.init(1 + 0.01 * rng.standard_normal(nn), u, -u, np.zeros(nn))
        s.step(steps, write_macro=True)
        return on_chip, [s.get_state()] + list(s.macro())


def same(monkeypatch, lat, args, steps, on_chip=True):
    a, got = state(monkeypatch, "", lat, args, steps)
    b, want = state(monkeypatch, "jit", lat, args, steps)
    assert a is on_chip and not b
    for x, y in zip(got, want):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("coll", [N.BGKW, N.TRT, N.MRT])
@pytest.mark.parametrize("shape", ["cavity", "channel"])
def test_reference_mode(monkeypatch, coll, shape):
    lat = lattice.cavity2d(143, 91) if shape == "cavity" else lattice.channel2d(197, 83, seed=3, size_scale=0.3)
    args = Arguments(u=0.05, viscosity=0.04, collision_model=coll, mode=N.MODE_REFERENCE, storage=N.STORE_F32,
                     init_equilibrium=1, outlet_profile=N.OUTLET_ZOUHE)
    same(monkeypatch, lat, args, 40)


# 152 tiles of 44 x 62 nodes, 2944 with their halo; the largest square; a square
# and a lattice just past them
@pytest.mark.parametrize("n,m,fits", [(352, 1178, True), (632, 632, True), (667, 613, False), (353, 1178, False)])
@pytest.mark.parametrize("storage", [N.STORE_F32, N.STORE_F16S])
def test_largest(monkeypatch, n, m, fits, storage):
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("sizes for 152 SMs")
    args = Arguments(u=0.1, viscosity=0.05, collision_model=N.MRT, mode=N.MODE_PHYSICS, storage=storage,
                     init_equilibrium=1, outlet_profile=N.OUTLET_ZOUHE)
    same(monkeypatch, lattice.cavity2d(n, m), args, 9, on_chip=fits)
