"""The staged kernels at the row lengths and value ranges where their paths
part: rows that are multiples of 4, 2 and 1 floats with a partial tile at the x
edge, down to one cell, and units that put density, pressure or slopes outside the range that the
shared reciprocals cover, everywhere or in some cells only, so that those faces
and quotients take the plain arithmetic.  Bitwise the oracle: one scheme, each
operation rounded the same."""
import numpy as np
import pytest

from nmhd_b200.problems import orszag_tang_3d
from oracle import oracle

from test_parity_gpu import assert_same, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(1, 5, 3), (2, 13, 7), (3, 5, 3), (4, 13, 7), (6, 5, 3), (34, 13, 7), (35, 13, 7), (36, 13, 7), (37, 9, 5), (64, 16, 8), (70, 18, 6),
                                      (100, 14, 6)])
@pytest.mark.parametrize("units", ["plain", "light", "light_mixed", "dense_mixed", "still"])
def test_staged_paths_match_oracle(gpu, nx, ny, nz, units):
    cfg, s = orszag_tang_3d(nx, ny=ny, nz=nz)
    rng = np.random.default_rng(nx)
    # density and pressure in units of `scale`, B in its root: the speeds stay
    scale = {"plain": 1.0, "light": 2.0 ** -46, "light_mixed": 2.0 ** -38, "dense_mixed": 2.0 ** 26, "still": 1.0}[units]
    s = s * np.array([scale, 1, 1, 1, scale] + [scale ** 0.5] * 3, np.float32).reshape(8, 1, 1, 1)
    # about 0.16 to 0.31 each: the mixed units put some cells on either side
    s[0] *= rng.uniform(0.7, 1.4, s[0].shape).astype(np.float32)
    s[4] *= rng.uniform(1.2, 2.3, s[4].shape).astype(np.float32)
    if units == "still":
        # v_z slopes that are not 0 but below 2^-74
        s[3] = (2.0 ** -80 * rng.uniform(-1, 1, s[3].shape)).astype(np.float32)
    s = np.ascontiguousarray(s, np.float32)
    o = oracle.proceed(cfg, s, 3)
    r = run_gpu(cfg, s, 3)
    assert np.isfinite(o["state"]).all()
    assert r["time"] == o["time"]
    assert_same(r["state"], o["state"])


@pytest.mark.parametrize("n", [(24, 20, 12), (32, 16, 8)])  # spacings that are no powers of two, and that are
@pytest.mark.parametrize("value", [np.nan, np.inf, -3e38])
@pytest.mark.parametrize("time_order", [1, 2])
def test_states_that_are_not_finite_spread_as_in_the_per_cell_kernels(gpu, n, value, time_order):
    """One value of one cell is not finite or overflows: the step ends in an error,
    and what it leaves is the per-cell kernels' state (the compiler's quotients and
    the plain limiter), NaN for NaN and infinity for infinity."""
    from nmhd_b200._lib import NmhdError
    from nmhd_b200.solver import MHDSolver
    for field in range(8):
        cfg, s = orszag_tang_3d(n[0], ny=n[1], nz=n[2])
        cfg.time_order = time_order
        s[field, 5, 9, 11] = value
        found = []
        for variant in (2, 5):
            with MHDSolver(cfg) as sol:
                sol.set_kernel(variant)
                sol.set_state(s)
                with pytest.raises(NmhdError):
                    sol.step(1)
                found.append(sol.get_state())
        assert np.array_equal(*found, equal_nan=True), (field, int((found[0] != found[1]).sum()))
