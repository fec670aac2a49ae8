"""The FP64 std chain evaluates each mutual pair once and still adds in one order: the default mode gives the
same bits in every run, whatever the cache of pair geometry holds."""

import numpy as np
import pytest

from test_gpu_parity import field_scale, fp64_tol

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "p", "c", "c11", "c12", "c13", "c22", "c23", "c33", "ax", "ay", "az", "du")


def std(ctx, wl, how):
    from sphexa_gb300 import sph
    ctx.set_params(ng0=int(wl.params["ng0"]), ngmax=int(wl.params["ngmax"]), bucket=int(wl.params["bucket"]),
                   minDt=float(wl.params["minDt"]))
    d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0")
    box = sph.Box(wl.box.copy(), wl.bc.copy())
    if how == "sweep":
        sph.sweep(ctx, d, box, "std")
    else:
        sph.Domain(ctx, box).sync(d)
        sph.find_neighbors_sfc(ctx, 0, wl.n, d)
        sph.compute_density(ctx, d)
        sph.compute_eos_hydro_std(ctx, d)
        sph.compute_iad(ctx, d)
        sph.compute_momentum_energy_std(ctx, d)
    out = {f: d.f[f].cpu().numpy() for f in FIELDS}
    out["minDt"] = np.float64(d.minDtCourant)
    return out


# warps and slices partly filled, 16 slices and fewer, one slice; few neighbours and lists cut at ngmax; more
# than 64 pairs of a particle owned by others
@pytest.mark.parametrize("n, ngmax", [(33, 150), (1331, 150), (20011, 150), (90001, 150), (330001, 150), (5003, 40),
                                      (4099, 400)])
def test_std_chain_gives_the_same_bits_in_every_run(n, ngmax):
    from sphexa_gb300 import sph, workloads as W
    wl = W.random_cube(n, seed=161 + n, periodic=n > 1000)
    rng = np.random.Generator(np.random.PCG64(162))
    wl.fields["m"] = (10.0 ** rng.uniform(-0.3, 0.3, n) / n).astype(np.float32).astype(np.float64)
    for k in ("vx", "vy", "vz"):
        wl.fields[k] = rng.normal(0.0, 0.2, n).astype(np.float32).astype(np.float64)
    if ngmax != 150:
        wl.params["ng0"], wl.params["ngmax"] = (30 if ngmax < 150 else 300), ngmax
    runs, fixed = [], None
    for arrays in (5, 5, 2, 0, 5):
        ctx = sph.Context(0)
        ctx.set_pair_cache(arrays)
        for how in ("sweep", "passes"):
            runs.append(std(ctx, wl, how))
        if fixed is None:
            ctx.set_deterministic(True)
            fixed = std(ctx, wl, "sweep")
        ctx.close()
    for r in runs[1:]:
        for f in (*FIELDS, "minDt"):
            assert np.array_equal(r[f], runs[0][f]), f
    for f in FIELDS:
        err = np.max(np.abs(runs[0][f] - fixed[f])) / field_scale(fixed, f)
        assert err <= fp64_tol(fixed, f, "std"), f"{f}: {err:.3e}"


def test_std_chain_without_room_for_records_walks_whole_lists():
    """On a nearly full device the passes fall back to the order-fixed walk (density and IAD are then its
    bits), with the same results to rounding."""
    from sphexa_gb300 import sph, workloads as W
    from test_gpu_pair_cache import MB, free_memory
    wl = W.random_cube(60000, seed=163, periodic=True)
    ctx = sph.Context(0)
    free = std(ctx, wl, "passes")
    ctx.close()
    ctx = sph.Context(0)
    ctx.set_deterministic(True)
    fixed = std(ctx, wl, "passes")
    ctx.close()
    ctx = sph.Context(0)
    ctx.set_pair_cache(0)
    d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0")
    box = sph.Box(wl.box.copy(), wl.bc.copy())
    sph.Domain(ctx, box).sync(d)
    sph.find_neighbors_sfc(ctx, 0, wl.n, d)
    with free_memory(400 * MB):  # the records need 36 bytes for about 55 pairs each, 120 MB: more than an eighth
        sph.compute_density(ctx, d)
        sph.compute_eos_hydro_std(ctx, d)
        sph.compute_iad(ctx, d)
        sph.compute_momentum_energy_std(ctx, d)
    for f in ("rho", "c11", "c23"):
        assert np.array_equal(d.f[f].cpu().numpy(), fixed[f]), f
    for f in FIELDS:
        err = np.max(np.abs(d.f[f].cpu().numpy() - free[f])) / field_scale(free, f)
        assert err <= 1e-12, f"{f}: {err:.3e}"
    ctx.close()
