"""Frozen neighbour lists with particles moved since the search, in periodic boxes: a pair across a face whose
owner's own 2h no longer reaches the face still counts at the other end."""

import numpy as np
import pytest

from test_gpu_parity import field_scale, fp64_tol

pytestmark = pytest.mark.gpu


def moved_set(ctx, n, chain, move=0.05):
    """a periodic set with h varied by 30 %, synced and searched, then moved by about `move` h"""
    import torch
    from sphexa_gb300 import sph, workloads as W
    wl = W.random_cube(n, seed=211, periodic=True)
    rng = np.random.Generator(np.random.PCG64(212))
    wl.fields["h"] = (wl.fields["h"] * np.exp(rng.normal(0.0, 0.3, n))).astype(np.float32).astype(np.float64)
    for k in ("vx", "vy", "vz"):
        wl.fields[k] = rng.normal(0.0, 0.2, n).astype(np.float32).astype(np.float64)
    ctx.set_params(ng0=100, ngmax=150, bucket=64, minDt=1e-3)
    d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0")
    box = sph.Box(wl.box.copy(), wl.bc.copy())
    sph.Domain(ctx, box).sync(d)
    sph.find_neighbors_sfc(ctx, 0, n, d)
    for k in ("x", "y", "z"):
        d.f[k].add_(move * d.f["h"] * torch.as_tensor(rng.normal(size=n), device="cuda:0"))
    return d


# fields whose sums take the particle's own kernel function only: there the order-fixed passes are right for any
# positions (each particle folds by its own 2h)
@pytest.mark.parametrize("arrays", [0, 5])
@pytest.mark.parametrize("n", [700, 4000, 30011])
@pytest.mark.parametrize("chain, fields", [("std", ("rho", "c11", "c12", "c33")),
                                           ("ve", ("xm", "kx", "gradh", "c11", "c12", "c33", "divv", "curlv"))])
def test_passes_on_moved_particles_match_the_order_fixed_form(gpu_ctx, chain, fields, n, arrays):
    from sphexa_gb300 import sph
    out = {}
    gpu_ctx.set_pair_cache(arrays)
    for det in (True, False):
        gpu_ctx.set_deterministic(False)
        d = moved_set(gpu_ctx, n, chain)
        gpu_ctx.set_deterministic(det)
        if chain == "std":
            sph.compute_density(gpu_ctx, d)
            sph.compute_eos_hydro_std(gpu_ctx, d)
            sph.compute_iad(gpu_ctx, d)
        else:
            sph.compute_xmass(gpu_ctx, d)
            sph.compute_ve_def_gradh(gpu_ctx, d)
            sph.compute_eos(gpu_ctx, d)
            sph.compute_iad_divv_curlv(gpu_ctx, d)
        out[det] = {f: d.f[f].cpu().numpy() for f in fields}
    gpu_ctx.set_deterministic(False)
    gpu_ctx.set_pair_cache(5)
    for f in fields:
        err = np.max(np.abs(out[False][f] - out[True][f])) / field_scale(out[True], f)
        assert err <= fp64_tol(out[True], f, chain), f"{f}: {err:.3e}"


@pytest.mark.parametrize("du", [False, True])
def test_std_adjoint_on_moved_particles_is_that_of_the_passes(du):
    """The gradient along a random direction against a central difference of the default passes (smooth kernel
    form; step 1e-6 of h: truncation 1e-12 of the third derivative's scale, rounding 1e-15 / 1e-6)."""
    import torch
    from sphexa_gb300 import autograd as AG, sph
    ctx = sph.Context(0)
    ctx.set_kernel_form(True)
    n = 4000
    d = moved_set(ctx, n, "std")
    sw = AG.FrozenStdSweep(ctx, d, None)
    vals = list(sw.inputs())
    rng = np.random.Generator(np.random.PCG64(213))
    out = sw.forward(*vals)
    w = [torch.as_tensor(rng.normal(size=n), device="cuda:0") / t.abs().max() for t in out]
    if not du:
        w[4] = torch.zeros_like(w[4])
    grads = sw.backward(*w)
    step = 1e-6 * vals[6]
    for q in range(3):
        dirn = step * torch.as_tensor(rng.normal(size=n), device="cuda:0")

        def loss(sign):
            moved = list(vals)
            moved[q] = vals[q] + sign * dirn
            return sum(float((a * b).sum()) for a, b in zip(w, sw.forward(*moved)))
        fd = 0.5 * (loss(1.0) - loss(-1.0))
        ad = float((grads[q] * dirn).sum())
        size = float((grads[q] * dirn).abs().sum())
        assert abs(ad - fd) <= 1e-6 * size, f"{q}: {ad:.9e} {fd:.9e} of {size:.3e}"
    ctx.close()
