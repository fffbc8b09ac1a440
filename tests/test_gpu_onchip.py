"""The on-chip multi-step kernel's handle: what happens beside the steps
themselves (which test_gpu_resident compares with the oracle)."""
import threading

import numpy as np
import pytest

from thesis_gb300 import lattice
from thesis_gb300 import native as N
from thesis_gb300.solver import Arguments, Solver

pytestmark = pytest.mark.gpu


def cavity(n, m, coll=N.MRT, mode=N.MODE_PHYSICS, storage=N.STORE_F32):
    return lattice.cavity2d(n, m), Arguments(u=0.1, viscosity=0.05, collision_model=coll, mode=mode, storage=storage,
                                             init_equilibrium=1, outlet_profile=N.OUTLET_ZOUHE)


def rest(nn):
    return np.ones(nn), np.zeros(nn), np.zeros(nn), np.zeros(nn)


def test_default_stream_busy():
    """Handles made and stepped while another thread keeps the default stream
    full: nothing of a handle's own clearing may wait behind that work."""
    import torch
    lat, args = cavity(256, 200)
    with Solver(lat, args) as s:
        s.init(*rest(lat.num_nodes))
        s.step(20)
        alone = s.get_state(), s.residual()[0]
    stop = threading.Event()

    def fill():
        a = torch.ones(2048, 2048, device="cuda")
        while not stop.is_set():
            for _ in range(20):
                a = a @ a * 0.0
            torch.cuda.synchronize()
    t = threading.Thread(target=fill)
    t.start()
    try:
        for _ in range(10):
            with Solver(lat, args) as s:
                s.init(*rest(lat.num_nodes))
                s.step(20)
                assert np.array_equal(s.get_state(), alone[0])
                assert s.residual()[0] == alone[1]
    finally:
        stop.set()
        t.join()
