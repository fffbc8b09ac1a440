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


def test_wait_that_gives_up():
    """A wait that runs out (one poll allowed) leaves the kernel at once; every
    reader and the next step report it, and a new state ends it."""
    lat, args = cavity(256, 200)
    nn = lat.num_nodes
    box = (0, 10, 0, 10, 0, 1)
    with Solver(lat, args) as s:
        assert s.on_chip
        s.init(*rest(nn))
        s.step(20)
        good = s.get_state()
        s.step(30)
        later = s.get_state()
        readers = [s.get_state, s.populations, s.macro, s.norms, s.residual, s.macro_diff, s.residual_l2,
                   s.residual_fd_rel_diff, lambda: s.momentum_exchange(box), lambda: s.step(1), lambda: s.step(20)]
        if (np.asarray(lat.bc[:, 5]) > 0).any():
            readers.append(lambda: s.reference_drag_lift(int(lat.bc[:, 5].max()), np.zeros(nn), np.zeros(nn)))
        for renew in (lambda: s.set_state(good), lambda: (s.init(*rest(nn)), s.step(20))):
            N.check(s._lib.lbm_test_on_chip(s._h, 0, 0, 0))
            s.step(30)
            for read in readers:
                with pytest.raises(N.LbmError) as e:
                    read()
                assert e.value.code == N.LBM_ERR_CUDA
            assert s.status == N.LBM_ERR_CUDA
            N.check(s._lib.lbm_test_on_chip(s._h, -1, 0, 0))
            renew()
            assert s.status == N.LBM_OK
            assert np.array_equal(s.get_state(), good)
            s.step(30)
            assert np.array_equal(s.get_state(), later)


def test_refused_launch():
    """A launch that the driver refuses (here: taken as refused) leaves the
    call to the launch-per-step kernel, with the same state and fields; the
    next call runs on chip again."""
    lat, args = cavity(256, 200)

    def run(refuse):
        with Solver(lat, args) as s:
            s.init(*rest(lat.num_nodes))
            for k in (20, 41, 7):
                N.check(s._lib.lbm_test_on_chip(s._h, -1, refuse, 0))
                s.step(k, write_macro=True)
            return [s.get_state()] + list(s.macro()) + [s.status]
    for a, b in zip(run(0), run(1)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n,m", [(13, 200), (61, 47), (203, 131), (400, 350)])
@pytest.mark.parametrize("storage", [N.STORE_F32, N.STORE_F16S])
def test_parts_of_the_chip(n, m, storage):
    """The cuts for a half, a quarter and an eighth of the SMs give the state
    of the cut for all of them (the last size fits no eighth)."""
    lat, args = cavity(n, m, storage=storage)

    def run(parts):
        with Solver(lat, args) as s:
            s.init(*rest(lat.num_nodes))
            N.check(s._lib.lbm_test_on_chip(s._h, -1, 0, parts))
            s.step(25)
            s.step(12, write_macro=True)
            return [s.get_state()] + list(s.macro())
    ref = run(1)
    for parts in (2, 4, 8):
        for a, b in zip(ref, run(parts)):
            assert np.array_equal(a, b)


def test_handles_side_by_side():
    """Six handles stepped by six threads on streams of their own, call after
    call, so that launches meet in flight: each ends as it does alone."""
    import torch
    cases = [cavity(128 + 8 * k, 96 + 40 * k, (N.BGKW, N.TRT, N.MRT)[k % 3]) for k in range(6)]

    def run(k, out):
        lat, args = cases[k]
        stream = torch.cuda.Stream()
        with Solver(lat, args) as s:
            s.init(*rest(lat.num_nodes))
            for _ in range(30):
                s.step(40, write_macro=False, stream=stream.cuda_stream)
            s.step(10, write_macro=True, stream=stream.cuda_stream)
            out[k] = [s.get_state()] + list(s.macro())
    alone, together = {}, {}
    for k in range(6):
        run(k, alone)
    threads = [threading.Thread(target=run, args=(k, together)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(6):
        for a, b in zip(alone[k], together[k]):
            assert np.array_equal(a, b)


def test_error_words_of_many_handles():
    """More handles at once than a page of error words holds: a wait that gives
    up in one is reported by that one alone, also after words were given back."""
    lat, args = cavity(24, 24)
    ss = [Solver(lat, args) for _ in range(1030)]
    try:
        for s in ss[::2]:
            s.close()
        ss = ss[1::2] + [Solver(lat, args) for _ in range(40)]
        for s in ss:
            s.init(*rest(lat.num_nodes))
        N.check(ss[7]._lib.lbm_test_on_chip(ss[7]._h, 0, 0, 0))
        for s in ss:
            s.step(10)
        for k, s in enumerate(ss):
            if k == 7:
                with pytest.raises(N.LbmError):
                    s.get_state()
            else:
                s.get_state()
    finally:
        for s in ss:
            s.close()


@pytest.mark.parametrize("n,m", [(96, 64), (250, 130)])
def test_tuning_keeps_steps_on_chip(n, m):
    """Handles of a tuned shape run on chip whatever kernel the tuning chose for
    a launch per step, and give the same state."""
    lat, args = cavity(n, m)

    def run(tune):
        with Solver(lat, args) as s:
            if tune:
                s.autotune(4)
            assert s.on_chip
            s.init(*rest(lat.num_nodes))
            s.step(30)
            return s.get_state()
    first = run(False)
    assert np.array_equal(first, run(True))
    assert np.array_equal(first, run(False))


def test_reductions_beside_a_busy_handle():
    """A handle that steps while another's launches are in flight reads its
    residuals without an error: that the other is not ready yet is none."""
    import torch
    big, bargs = cavity(600, 600)
    lat, args = cavity(96, 80)
    stream = torch.cuda.Stream()
    with Solver(big, bargs) as b, Solver(lat, args) as s:
        b.init(*rest(big.num_nodes))
        s.init(*rest(lat.num_nodes))
        for _ in range(3):
            b.step(4000, write_macro=False, stream=stream.cuda_stream)
            s.step(8)
            assert np.isfinite(s.residual()[0])
            assert np.isfinite(s.macro_diff()[0]).all()
            assert np.isfinite(s.residual_l2()[0])


def test_calls_of_several_launches(monkeypatch):
    """A call longer than a launch holds (512 steps), and one step longer, gives
    the state of a launch per step."""
    lat, args = cavity(70, 45)

    def run():
        with Solver(lat, args) as s:
            s.init(*rest(lat.num_nodes))
            s.step(513)
            s.step(1100, write_macro=True)
            return [s.get_state()] + list(s.macro())
    got = run()
    monkeypatch.setenv("THESIS_LBM_KERNEL", "jit")
    for a, b in zip(got, run()):
        assert np.array_equal(a, b)
