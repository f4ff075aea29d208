"""States whose fields lie one after another in memory: one copy only inside one
allocation."""
import ctypes
import mmap

import numpy as np
import pytest

from nmhd_b200 import _lib
from nmhd_b200.problems import orszag_tang_3d

from test_face_math_cpu import lib

PAGE = 4096


def one_run(fields, n, allocations, known=True):
    c = lambda v: (ctypes.c_size_t * max(1, len(v)))(*v)
    return bool(lib().cellh_one_run(c(fields), ctypes.c_long(n), c([a for a, _ in allocations]),
                                    c([b for _, b in allocations]), len(allocations), int(known)))


def test_fields_are_copied_as_one_only_inside_one_allocation():
    n, size, at = 1024, PAGE, 1 << 20
    row = [at + v * size for v in range(8)]
    end = row[-1] + size
    assert one_run(row, n, [(at, end)])
    assert one_run(row, n, [(at - size, end + size)])
    assert one_run(row, n, [])  # pageable
    # eight allocations back to back, two, and a pinned one amid pageable memory
    assert not one_run(row, n, [(r, r + size) for r in row])
    assert not one_run(row, n, [(at, row[5]), (row[5], end)])
    assert not one_run(row, n, [(row[3], row[4])])
    assert not one_run(row, n, [(at, end - 4)])
    assert not one_run(row, n, [(at, end)], known=False)
    # a gap, another order, a field of its own
    assert not one_run(row[:7] + [end], n, [(at, end + size)])
    assert not one_run(row[::-1], n, [(at, end)])
    assert not one_run([at] * 8, n, [(at, end)])


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", ["none", "each", "all", "one"])
def test_states_in_buffers_pinned_one_by_one(gpu, pinned):
    """Eight page-aligned fields back to back, each pinned by itself."""
    import torch
    from nmhd_b200.batch import BatchSolver
    from nmhd_b200.solver import MHDSolver
    cfg, s = orszag_tang_3d(32, ny=16, nz=8)
    size = 4 * cfg.cells
    assert size % PAGE == 0
    buf = mmap.mmap(-1, 8 * size)
    host = np.frombuffer(buf, np.float32).reshape((8,) + cfg.shape)
    base = host.ctypes.data
    cudart = torch.cuda.cudart()
    spans = {"none": [], "each": [(base + v * size, size) for v in range(8)], "all": [(base, 8 * size)],
             "one": [(base + 2 * size, size)]}[pinned]
    for at, length in spans:
        assert int(cudart.cudaHostRegister(at, length, 0)) == 0
    try:
        ptrs = (ctypes.c_void_p * 8)(*[base + v * size for v in range(8)])
        with MHDSolver(cfg) as one, BatchSolver([cfg, cfg]) as batch:
            for handle, put, get in ((one._h, _lib.lib().nmhd_set_state, _lib.lib().nmhd_get_state),
                                     (batch._h, lambda h, p, d: _lib.lib().nmhd_batch_set_state(h, 1, p, d),
                                      lambda h, p, d: _lib.lib().nmhd_batch_get_state(h, 1, p, d))):
                host[:] = s
                assert put(handle, ptrs, 0) == 0
                host[:] = 0
                assert get(handle, ptrs, 0) == 0
                assert np.array_equal(host, s)
    finally:
        for at, _ in spans:
            cudart.cudaHostUnregister(at)
