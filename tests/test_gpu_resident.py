"""On-chip multi-step kernel (2D lattices whose populations fit the SMs'
shared memory, many steps per launch) against the oracle, with the tolerances
of test_gpu_parity, at the sizes where its tiling can go wrong: one tile, one
row or column of tiles, uneven tiles, wrapped tile neighbours, the largest
lattice that fits; and against the launch-per-step kernel over several calls."""
import numpy as np
import pytest

from test_gpu_parity import compare, run_pair
from thesis_gb300 import lattice
from thesis_gb300 import native as N
from thesis_gb300.lattice import Lattice
from thesis_gb300.solver import Arguments, Solver

pytestmark = pytest.mark.gpu


def cavity(n, m, coll, mode, storage):
    return lattice.cavity2d(n, m), Arguments(u=0.1, viscosity=0.05, collision_model=coll, mode=mode, storage=storage,
                                             init_equilibrium=1, outlet_profile=N.OUTLET_ZOUHE)


def rest(nn):
    return np.ones(nn), np.zeros(nn), np.zeros(nn), np.zeros(nn)


@pytest.mark.parametrize("n,m", [(3, 3), (96, 1), (1, 97), (2, 130), (191, 2), (61, 47), (128, 128), (1031, 37),
                                 (667, 613)])
@pytest.mark.parametrize("coll,mode,storage", [(N.BGKW, N.MODE_REFERENCE, N.STORE_F32),
                                               (N.TRT, N.MODE_PHYSICS, N.STORE_F32),
                                               (N.MRT, N.MODE_PHYSICS, N.STORE_F16S)])
def test_cavity_sizes(oracle, n, m, coll, mode, storage):
    if storage == N.STORE_F16S and (n < 3 or m < 2):
        pytest.skip("no flow (every lid node is a corner): F16S is compared by relative errors of it")
    lat, args = cavity(n, m, coll, mode, storage)
    g, r, fl = run_pair(oracle, lat, args, 9, init=rest(lat.num_nodes))
    compare(g, r, fl, storage, 2)


@pytest.mark.parametrize("n,m", [(7, 5), (96, 1), (1, 97), (96, 3), (130, 61), (300, 301)])
@pytest.mark.parametrize("periodic", [(1, 1, 0), (1, 0, 0)])
def test_periodic_with_solids(oracle, n, m, periodic):
    rng = np.random.default_rng(n)
    fluid = (rng.random(n * m) > 0.1).astype(np.int32)
    lat = Lattice(2, n, m, 1, fluid)
    args = Arguments(viscosity=0.06, collision_model=N.MRT, mode=N.MODE_PHYSICS, init_equilibrium=1, periodic=periodic)
    u = np.where(fluid, 0.05 * rng.standard_normal(n * m), 0.0)
    init = (1 + 0.01 * rng.standard_normal(n * m), u, -u, np.zeros(n * m))
    g, r, fl = run_pair(oracle, lat, args, 11, init=init)
    compare(g, r, fl, N.STORE_F32, 2)


def test_channel_inlet_outlet(oracle):
    lat = lattice.channel2d(260, 66, seed=3, size_scale=0.25)
    args = Arguments(u=0.05, viscosity=0.03, collision_model=N.TRT, mode=N.MODE_PHYSICS, init_equilibrium=1,
                     outlet_profile=N.OUTLET_PRESSURE, rho_out=1.0)
    g, r, fl = run_pair(oracle, lat, args, 30, init=rest(lat.num_nodes))
    compare(g, r, fl, N.STORE_F32, 2)


@pytest.mark.parametrize("storage", [N.STORE_F32, N.STORE_F16S])
def test_calls_of_several_lengths(monkeypatch, storage):
    """Calls shorter than, equal to and longer than the shortest run kept on
    chip, on the handle's stream and on another one, give the state that a
    launch per step gives: the node arithmetic is the same code, so only the
    contraction of a multiply-add may differ (one rounding, 2^-24 of w_d, per
    operation and step; FP16 storage keeps 2^-11 of the deviation)."""
    import torch
    lat, args = cavity(203, 87, N.MRT, N.MODE_PHYSICS, storage)
    calls = [1, 4, 3, 5, 40, 2]

    def run():
        stream = torch.cuda.Stream()
        with Solver(lat, args) as s:
            s.init(*rest(lat.num_nodes))
            for k, c in enumerate(calls):
                s.step(c, write_macro=True, stream=stream.cuda_stream if k == 4 else None)
                torch.cuda.synchronize()
            return s.populations(), s.macro()
    f, mac = run()
    monkeypatch.setenv("THESIS_LBM_KERNEL", "jit")
    f1, mac1 = run()
    tol = 55 * 20 * 2.0 ** -24 * 0.45 if storage == N.STORE_F32 else 5e-3 * np.abs(f1 - f1.mean(1, keepdims=True)).max()
    assert np.abs(f - f1).max() <= tol
    for a, b in zip(mac[:3], mac1[:3]):
        assert np.abs(a - b).max() <= 9 * tol


def test_handles_of_two_threads():
    """Two threads step their own lattices at the same time, each lattice as
    wide as the GPU: every launch runs to its end and gives the state of a run
    alone."""
    import threading
    cases = [cavity(512, 300, N.MRT, N.MODE_PHYSICS, N.STORE_F32), cavity(300, 400, N.BGKW, N.MODE_REFERENCE, N.STORE_F32)]
    out = {}

    def run(k, tag):
        lat, args = cases[k]
        with Solver(lat, args) as s:
            s.init(*rest(lat.num_nodes))
            for _ in range(20):
                s.step(50)
            s.step(10, write_macro=True)
            out[tag, k] = s.get_state(), s.macro()
    for k in range(2):
        run(k, "alone")
    threads = [threading.Thread(target=run, args=(k, "together")) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert np.array_equal(out["alone", k][0], out["together", k][0])
        for a, b in zip(out["alone", k][1], out["together", k][1]):
            assert np.array_equal(a, b)
