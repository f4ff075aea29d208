"""The fast-arithmetic flag's results, pinned.

Its kernel is compiled with contraction and approximate division and square
root, so no restatement of it is bitwise, and a change of its formulas shows in no
other test: rounding-size differences grow to 5e-4 within 16 steps.  The digests
below are those of the reference's expressions in its order, each quotient and root
the compiler's own.  They hold for the compiler of this repository (CUDA 12.9);
with another one, measure the mode's error against an FP64 run before taking new
digests."""
import hashlib

import pytest

from nmhd_b200.config import FLAG_FAST_ARITHMETIC
from nmhd_b200.problems import orszag_tang_3d, shearing_box
from nmhd_b200.solver import MHDSolver

pytestmark = pytest.mark.gpu

DIGESTS = {
    "mri": "96e7e1ad2f4e76aa",
    "ragged": "b83c0442cf262317",
    "vortex": "91cfa3c386361257",
    "order1": "ab01568fe4565c90",
    "weak_field": "b305f434a7b8a37c",
}


@pytest.mark.parametrize("case", sorted(DIGESTS))
def test_fast_arithmetic_bits(gpu, case):
    if case == "vortex":
        cfg, s = orszag_tang_3d(36, ny=20, nz=12)
    elif case == "ragged":  # rows of pairs, spacings that are no powers of two
        cfg, s = shearing_box(n_radial=27, n_azimuthal=50, n_vertical=11, l_azimuthal=2.5, l_vertical=0.6, seed=5)
    else:
        cfg, s = shearing_box(n_radial=32, n_azimuthal=64, n_vertical=16, l_azimuthal=4.0, seed=7)
        if case == "order1":
            cfg.space_order = 1
        if case == "weak_field":  # slopes whose products underflow
            s[5:8] *= 1e-20
    cfg.flags = FLAG_FAST_ARITHMETIC
    with MHDSolver(cfg) as sol:
        sol.set_state(s)
        sol.step(8)
        state = sol.get_state()
    assert hashlib.sha256(state.tobytes()).hexdigest()[:16] == DIGESTS[case]
