"""The switch between density sums that keep their rounding errors (sets in 16 slices: up to 648 warps, 20,736
particles) and plain ones, and the Courant time step of the two summation modes."""

import numpy as np
import pytest

from test_gpu_parity import field_scale, fp64_tol, run_gpu

pytestmark = pytest.mark.gpu

FIELDS = ("xm", "kx", "gradh")


def test_largest_set_with_kept_rounding_errors(gpu_ctx):
    """20,736 particles: hi + lo carries each sum to about 1e-32 of it in any order, so that runs differ only where
    it lies that close to the middle of two numbers (one sum in 1e15)."""
    from sphexa_gb300 import workloads as W
    wl = W.random_cube(20736, seed=181, periodic=False)
    gpu_ctx.set_deterministic(False)
    a, b = run_gpu(gpu_ctx, wl, "ve", False), run_gpu(gpu_ctx, wl, "ve", False)
    for f in FIELDS:
        assert np.array_equal(a[f], b[f]), f


@pytest.mark.parametrize("n", [20736, 20737])
def test_both_sides_of_the_switch_match_the_order_fixed_sums(gpu_ctx, n):
    from sphexa_gb300 import workloads as W
    wl = W.random_cube(n, seed=182, periodic=False)
    out = {}
    for det in (True, False):
        gpu_ctx.set_deterministic(det)
        out[det] = run_gpu(gpu_ctx, wl, "ve", False)
    gpu_ctx.set_deterministic(False)
    for f in FIELDS:
        err = np.max(np.abs(out[False][f] - out[True][f])) / field_scale(out[True], f)
        assert err <= fp64_tol(out[True], f, "ve"), f"{f}: {err:.3e}"


@pytest.mark.parametrize("arrays", [0, 2, 5])
def test_ve_courant_step_is_that_of_the_order_fixed_passes(gpu_ctx, arrays):
    """Without cleaning every FP64 form of the VE momentum-energy pass forms r.v and the signal velocity in one
    order of FMAs: the time steps of both modes agree bit for bit."""
    from sphexa_gb300 import workloads as W
    wl = W.fourier(15, seed=183, rho_seed=184, v_seed=185)
    gpu_ctx.set_pair_cache(arrays)
    dt = []
    for det in (True, False):
        gpu_ctx.set_deterministic(det)
        dt.append(run_gpu(gpu_ctx, wl, "ve", False)["minDt"])
    gpu_ctx.set_deterministic(False)
    gpu_ctx.set_pair_cache(5)
    assert dt[0] == dt[1]
