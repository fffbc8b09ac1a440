"""Steps replayed from captured graphs (lattices that do not run on chip) and
steps recorded into a caller's own capture, against steps launched one by one:
the same bits."""
import numpy as np
import pytest

from thesis_gb300 import lattice
from thesis_gb300 import native as N
from thesis_gb300.solver import Arguments, Solver

pytestmark = pytest.mark.gpu


def solver(h, storage):
    lat = lattice.cavity3d(20, 18, h) if h > 1 else lattice.cavity2d(24, 20)
    args = Arguments(u=0.1, viscosity=0.1, collision_model=N.MRT, mode=N.MODE_PHYSICS, storage=storage,
                     init_equilibrium=1, outlet_profile=N.OUTLET_ZOUHE)
    s = Solver(lat, args)
    nn = lat.num_nodes
    s.init(np.ones(nn), np.zeros(nn), np.zeros(nn), np.zeros(nn))
    return s


def result(s):
    return [s.populations()] + list(s.macro())


def single(h, storage, steps):
    with solver(h, storage) as s:
        for k in range(steps):
            s.step(1, write_macro=k == steps - 1)
        return result(s)


# calls around the shortest that take the two-step and the sixteen-step graph,
# with odd and even remainders, from both buffers
@pytest.mark.parametrize("calls", [(8,), (9, 9, 10), (32, 33), (33, 34, 41), (48, 57, 23), (7, 80, 1, 31)])
@pytest.mark.parametrize("h,storage", [(16, N.STORE_F32), (16, N.STORE_F16S), (1, N.STORE_F64)])
def test_replayed_steps(h, storage, calls):
    with solver(h, storage) as s:
        assert not s.on_chip
        for k, c in enumerate(calls):
            s.step(c, write_macro=k % 2 == 1 or k == len(calls) - 1)
        got = result(s)
    for a, b in zip(got, single(h, storage, sum(calls))):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("h,storage", [(1, N.STORE_F32), (1, N.STORE_F16S), (16, N.STORE_F32)])
@pytest.mark.parametrize("steps", [2, 6, 40])
def test_captured_steps(h, storage, steps):
    """A call on a stream under capture records its steps; an even number
    leaves the buffers as they were, so the graph can be replayed."""
    import torch
    with solver(h, storage) as s:
        stream = torch.cuda.Stream()
        s.step(10)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            s.step(steps, write_macro=True, stream=stream.cuda_stream)
        g.replay()
        g.replay()
        torch.cuda.synchronize()
        got = result(s)
    for a, b in zip(got, single(h, storage, 10 + 2 * steps)):
        assert np.array_equal(a, b)
