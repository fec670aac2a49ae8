"""Periodic lattices of a few particles a side, whose pairs lie at exactly half the box."""

import numpy as np
import pytest

from test_gpu_parity import field_scale, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [0.55, 0.6, 0.7])
def test_mixed_std_pairs_at_half_the_box(gpu_ctx, radius):
    """A 4^3 lattice with 2h between 1/2 and 3/4 of the box: both images of a pair at half the box are equally
    near, and r_ij = -r_ji as in the FP64 form (which folds beyond 2h).  FP32 arithmetic: 1e-5 of the field."""
    from sphexa_gb300 import workloads as W
    wl = W.random_cube(64, seed=221, periodic=True)
    g = np.stack(np.meshgrid(*[(np.arange(4) + 0.5) / 4] * 3, indexing="ij")).reshape(3, -1)
    for k, q in zip("xyz", g):
        wl.fields[k] = q.copy()
    rng = np.random.Generator(np.random.PCG64(222))
    wl.fields["h"][:] = np.float32(radius / 2)
    wl.fields["m"] = (rng.uniform(0.5, 1.5, 64) / 64).astype(np.float32).astype(np.float64)
    for k in ("vx", "vy", "vz"):
        wl.fields[k] = rng.normal(0.0, 0.2, 64).astype(np.float32).astype(np.float64)
    gpu_ctx.set_deterministic(True)
    ref = run_gpu(gpu_ctx, wl, "std", False, "fp64")
    gpu_ctx.set_deterministic(False)
    r = run_gpu(gpu_ctx, wl, "std", False, "mixed")
    np.testing.assert_array_equal(r["nc"], ref["nc"])
    for f in ("rho", "c11", "c12", "c13", "c22", "c23", "c33", "ax", "ay", "az", "du"):
        err = np.max(np.abs(r[f] - ref[f])) / field_scale(ref, f)
        assert err <= 1e-5, f"{f}: {err:.3e}"
