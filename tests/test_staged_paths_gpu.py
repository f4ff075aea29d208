"""The staged kernels at the row lengths and value ranges where their paths
part: rows that are multiples of 4, 2 and 1 floats with a partial tile at the x
edge, down to one cell, and units that put density, pressure or slopes outside the range that the
shared reciprocals cover, everywhere or in some cells only, so that those faces
and quotients take the plain arithmetic.  Bitwise the oracle: one scheme, each
operation rounded the same."""
import numpy as np
import pytest

from nmhd_b200.problems import orszag_tang_3d, shearing_box
from nmhd_b200.solver import MHDSolver
from oracle import oracle

from test_parity_gpu import assert_same, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(1, 5, 3), (2, 13, 7), (3, 5, 3), (4, 13, 7), (6, 5, 3), (34, 13, 7),
                                      (35, 13, 7), (36, 13, 7), (37, 9, 5), (64, 16, 8), (70, 18, 6), (100, 14, 6),
                                      # more tiles than SMs: a CTA takes a tile's three axes
                                      (100, 34, 24), (102, 34, 24), (101, 34, 24),
                                      # 1,105 tiles: the clock advances in a kernel of its own
                                      (130, 50, 34)])
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


@pytest.mark.parametrize("extent", [3e-13, 5e12])
def test_spacings_out_of_range_match_oracle(gpu, extent):
    """Spacings below 2^-40 and above 2^30, which only the update divides by."""
    cfg, s = orszag_tang_3d(36, ny=14, nz=6, extent=extent)
    o = oracle.proceed(cfg, s, 3)
    r = run_gpu(cfg, s, 3)
    assert np.isfinite(o["state"]).all()
    assert r["time"] == o["time"]
    assert_same(r["state"], o["state"])


def test_faces_out_of_range_are_not_solved_twice(gpu):
    """Density and pressure, or the field, in units that the shared reciprocals do
    not cover: the faces take the plain arithmetic alone, 1.4 times the usual launch
    and not 2.3."""
    cfg, s = shearing_box(n_radial=64, n_azimuthal=128, n_vertical=64)
    times = {}
    for units, scale in (("usual", [1.0, 1.0]), ("light", [2.0 ** -46, 2.0 ** -23]), ("weak", [1.0, 1e-18])):
        w = s.copy()
        w[[0, 4]] *= np.float32(scale[0])
        w[5:8] *= np.float32(scale[1])
        with MHDSolver(cfg) as sol:
            sol.set_state(w)
            sol.step(4)
            times[units] = min(sol.profile(4)["flux_stage1"][0] for _ in range(5))
    assert times["light"] < 1.8 * times["usual"] and times["weak"] < 1.8 * times["usual"], times
