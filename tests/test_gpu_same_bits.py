"""Every storage-unit kernel form of a lattice gives the same bits: the
default choice, one node per thread, walks along z, two z nodes on packed
FP32x2, the batch and the on-chip kernel share their node arithmetic, whose
roundings are written out.  Block and walk choices follow the extents, so the
extents here sit around them (rows that fill blocks of 64, 96, 160 threads or
leave lanes idle, columns that end inside a walk)."""
import numpy as np
import pytest

from thesis_gb300 import lattice
from thesis_gb300 import native as N
from thesis_gb300.batch import Batch
from thesis_gb300.solver import Arguments, Solver

pytestmark = pytest.mark.gpu


def state(monkeypatch, kernel, lat, args, steps):
    if kernel:
        monkeypatch.setenv("THESIS_LBM_KERNEL", kernel)
    else:
        monkeypatch.delenv("THESIS_LBM_KERNEL", raising=False)
    nn = lat.num_nodes
    with Solver(lat, args) as s:
        s.init(np.ones(nn), np.zeros(nn), np.zeros(nn), np.zeros(nn))
        s.step(steps)
        return s.get_state()


@pytest.mark.parametrize("shape", [(64, 64, 49), (96, 96, 110), (75, 61, 47), (150, 90, 75), (33, 100, 65)])
@pytest.mark.parametrize("coll", [N.BGKW, N.TRT, N.MRT])
@pytest.mark.parametrize("storage", [N.STORE_F32, N.STORE_F16S])
def test_duct(monkeypatch, shape, coll, storage):
    lat = lattice.sphere_duct(*shape, porosity=0.8, rmin=4, rmax=8, seed=2)
    args = Arguments(viscosity=0.1, collision_model=coll, mode=N.MODE_PHYSICS, storage=storage, init_equilibrium=1,
                     inlet_profile=N.INLET_PRESSURE, outlet_profile=N.OUTLET_PRESSURE, rho_in=1.005, rho_out=1.0)
    want = state(monkeypatch, "jith", lat, args, 20)
    for kernel in ("", "jithz3b96m12", "jithz4b64m10q"):
        assert np.array_equal(state(monkeypatch, kernel, lat, args, 20), want), kernel


@pytest.mark.parametrize("coll", [N.BGKW, N.TRT, N.MRT])
@pytest.mark.parametrize("storage", [N.STORE_F32, N.STORE_F16S])
def test_channel(monkeypatch, coll, storage):
    lat = lattice.channel2d(197, 83, seed=3, size_scale=0.3)
    args = Arguments(u=0.05, viscosity=0.03, collision_model=coll, mode=N.MODE_PHYSICS, storage=storage,
                     init_equilibrium=1, outlet_profile=N.OUTLET_PRESSURE, rho_out=1.0)
    want = state(monkeypatch, "jith", lat, args, 20)
    assert np.array_equal(state(monkeypatch, "", lat, args, 20), want)
    nn = lat.num_nodes
    z = np.zeros(nn)
    with Solver(lat, args) as s, Batch([lat, lat], [args, args]) as b:
        s.init(np.ones(nn), z, z, z)
        s.step(20)
        b.init()
        for d in range(2):
            b.init_fields(d, np.ones(nn), z, z, z)
        b.step(20)
        for d in range(2):
            assert np.array_equal(b.populations(d), s.populations())


@pytest.mark.parametrize("periodic", [(1, 1, 1), (0, 1, 0)])
@pytest.mark.parametrize("storage", [N.STORE_F32, N.STORE_F16S])
@pytest.mark.parametrize("dims", [2, 3])
def test_batch_sizes(monkeypatch, periodic, storage, dims):
    """Domains around the batch's tiles (32 nodes by an even number of rows):
    one row, odd rows, pairs that wrap, scattered solids; three dimensions,
    where rows of a tile span planes."""
    monkeypatch.setenv("THESIS_LBM_KERNEL", "jith")
    rng = np.random.default_rng(4)
    shapes = [(31, 1, 1), (32, 2, 1), (33, 3, 1), (65, 37, 1), (130, 64, 1)] if dims == 2 else [(20, 10, 7), (33, 5, 3)]
    lats, args, starts = [], [], []
    for n, m, h in shapes:
        nn = n * m * h
        fluid = (rng.random(nn) > 0.1).astype(np.int32)
        lats.append(lattice.Lattice(dims, n, m, h, fluid))
        args.append(Arguments(viscosity=0.06, collision_model=N.MRT, mode=N.MODE_PHYSICS, init_equilibrium=1,
                              storage=storage, periodic=periodic))
        u = np.where(fluid, 0.05 * rng.standard_normal(nn), 0.0)
        starts.append((1 + 0.01 * rng.standard_normal(nn), u, -u, np.zeros(nn)))
    with Batch(lats, args) as b:
        b.init()
        for d, st in enumerate(starts):
            b.init_fields(d, *st)
        b.step(17)
        got = [b.populations(d) for d in range(len(lats))]
    for lat, a, st, f in zip(lats, args, starts, got):
        with Solver(lat, a) as s:
            s.init(*st)
            s.step(17)
            want = s.populations()
        fl = lat.node_type == 1
        assert np.array_equal(f[:, fl], want[:, fl])


@pytest.mark.parametrize("coll", [N.BGKW, N.TRT, N.MRT])
@pytest.mark.parametrize("storage", [N.STORE_F32, N.STORE_F16S])
@pytest.mark.parametrize("domains,n,m", [(1, 40, 40), (8, 256, 256), (12, 192, 192), (3, 1024, 256)])
def test_batch_forms(monkeypatch, coll, storage, domains, n, m):
    """The forms of the D2Q9 batch kernel (blocks per SM, chosen by the active
    domains' tiles: five, five, six, and seven for channels), and a batch that
    goes from form to form as domains retire between replayed calls."""
    channel = n != m
    lat = lattice.channel2d(n, m, seed=2) if channel else lattice.cavity2d(n)
    args = Arguments(u=0.05, viscosity=0.05, collision_model=coll, mode=N.MODE_PHYSICS, storage=storage,
                     init_equilibrium=1, outlet_profile=N.OUTLET_PRESSURE if channel else N.OUTLET_ZOUHE, rho_out=1.0)
    nn = lat.num_nodes
    z = np.zeros(nn)
    monkeypatch.setenv("THESIS_LBM_KERNEL", "jith")
    with Solver(lat, args) as s, Batch([lat] * domains, [args] * domains) as b:
        s.init(np.ones(nn), z, z, z)
        b.init()
        for d in range(domains):
            b.init_fields(d, np.ones(nn), z, z, z)
        s.step(20)
        first = s.populations()
        s.step(20)
        second = s.populations()
        b.step(20)
        b.set_active([int(d == 0 or d % 3 > 0) for d in range(domains)])
        b.step(20)
        for d in range(domains):
            assert np.array_equal(b.populations(d), second if d == 0 or d % 3 > 0 else first)
