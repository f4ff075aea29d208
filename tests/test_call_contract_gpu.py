"""What nmhd.h promises of every call: it returns when its work is done, on any
thread, and the clock that the host knows is the device's."""
import ctypes
import math

import numpy as np
import pytest

from nmhd_b200 import _lib
from nmhd_b200.problems import orszag_tang_3d, shearing_box
from nmhd_b200.slab import slab_config
from nmhd_b200.solver import MHDSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["set_time", "set_state", "set_state_device", "slab_begin", "get_state"])
def test_calls_return_when_the_stream_is_done(gpu, call):
    import torch
    cfg, s = shearing_box(n_radial=16, n_azimuthal=32, n_vertical=8, l_azimuthal=4.0)
    if call == "slab_begin":
        cfg = slab_config(cfg, 2)
        s = np.ascontiguousarray(s[:, :, :cfg.size_y])
    stream = torch.cuda.Stream(device=gpu)
    with MHDSolver(cfg) as sol:
        sol.set_stream(stream.cuda_stream)
        sol.set_state(s)
        on_device = torch.from_numpy(s).to(gpu)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)  # about 10 ms
        assert not stream.query()
        if call == "set_time":
            sol.set_time(0.25, 3)
        elif call == "set_state":
            sol.set_state(s)
        elif call == "set_state_device":
            sol.set_state_device(on_device)
        elif call == "slab_begin":
            assert _lib.lib().nmhd_slab_begin(sol._h, math.inf) == 0
        else:
            assert np.array_equal(sol.get_state(), s)
        assert stream.query()
        sol.set_stream(None)


def test_calls_from_a_thread_whose_device_is_another(gpu):
    """The copies and graph launches of these calls need no current device; the
    control block's write must not either."""
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("one GPU")
    cfg, s = orszag_tang_3d(16)
    with MHDSolver(cfg) as sol, MHDSolver(cfg) as ref:
        for x in (sol, ref):
            x.set_state(s)
            x.prepare(4)
            x.step(4)
        ref.step(4)
        with torch.cuda.device(1):
            sol.step(4)
            assert torch.cuda.current_device() == 1
            state, clock = sol.get_state(), sol.current_time()
            sol.set_time(0.5, 7)
            sol.set_state(s)
            assert torch.cuda.current_device() == 1
        assert clock == ref.current_time() and np.array_equal(state, ref.get_state())
        assert sol.current_time() == 0.5 and sol.generation() == 7


def test_host_clock_is_the_devices_whatever_the_order_of_calls(gpu):
    """Every call that moves the clock, in seeded orders, against a solver whose
    control block is read back from the device each time (nmhd_cfl_slot, whose
    holder may write it, turns the host's copy off)."""
    cfg, s = shearing_box(n_radial=16, n_azimuthal=32, n_vertical=8, l_azimuthal=4.0, seed=9)
    rng = np.random.default_rng(11)
    with MHDSolver(cfg) as sol, MHDSolver(cfg) as ref:
        assert _lib.lib().nmhd_cfl_slot(ref._h)
        for x in (sol, ref):
            x.set_state(s)

        calls = [lambda x: x.step(3), lambda x: x.proceed(math.inf, 30.0, 2), lambda x: x.proceed(x.current_time() + 0.02),
                 lambda x: x.set_time(0.125, 40), lambda x: x.set_state(s), lambda x: x.profile(2) and None,
                 lambda x: x.loss_run(3) and None, lambda x: x.adjoint(2)[0], lambda x: x.step(20)]
        for k in rng.integers(0, len(calls), 40):
            a, b = calls[k](sol), calls[k](ref)
            assert a is b or a == b
            assert sol.current_time() == ref.current_time() and sol.generation() == ref.generation()
            assert np.array_equal(sol.get_state(), ref.get_state())
        sol.autotune(steps=1)
        assert sol.current_time() == ref.current_time() and sol.generation() == ref.generation()
        assert np.array_equal(sol.get_state(), ref.get_state())
        sol.step(2)
        ref.step(2)
        assert sol.current_time() == ref.current_time() and np.array_equal(sol.get_state(), ref.get_state())
        # a state that is not valid, and what follows it
        bad = s.copy()
        bad[4] = -1.0
        for x in (sol, ref):
            x.set_state(bad)
            with pytest.raises(_lib.NmhdError):
                x.step(3)
            with pytest.raises(_lib.NmhdError):
                x.step(1)
        assert sol.generation() == ref.generation()
        for x in (sol, ref):
            x.set_state(s)
            x.set_time(0.0, 0)  # the failed step's time may be NaN
            x.step(2)
        assert sol.current_time() == ref.current_time() and np.array_equal(sol.get_state(), ref.get_state())
