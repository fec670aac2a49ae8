"""The FP64 pass variants with inputs near the ends of their types' range: the one-evaluation form of each
mutual pair against the order-fixed form on the same inputs, and neighbour counts against the oracle."""

import numpy as np
import pytest

from test_gpu_parity import field_scale, fp64_tol, run_gpu

pytestmark = pytest.mark.gpu

ME_FIELDS = ("ax", "ay", "az", "du")


def momentum_energy_both(gpu_ctx, edit, clean=False, side=12, seed=111):
    """du, ax, ay, az and the time step of the default and the order-fixed momentum-energy pass after
    edit(d) changed fields of a jittered lattice that went through the passes before it"""
    from sphexa_gb300 import sph, workloads as W
    wl = W.fourier(side, seed=seed, rho_seed=seed + 1, v_seed=seed + 2)
    out = {}
    for det in (True, False):
        gpu_ctx.set_deterministic(det)
        gpu_ctx.set_params(ng0=int(wl.params["ng0"]), ngmax=int(wl.params["ngmax"]), bucket=int(wl.params["bucket"]),
                           minDt=float(wl.params["minDt"]))
        d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0", av_clean=clean)
        box = sph.Box(wl.box.copy(), wl.bc.copy())
        sph.Domain(gpu_ctx, box).sync(d)
        sph.find_neighbors_sfc(gpu_ctx, 0, wl.n, d)
        gpu_ctx.set_deterministic(True)  # the same inputs of the last pass for both forms
        sph.compute_xmass(gpu_ctx, d)
        sph.compute_ve_def_gradh(gpu_ctx, d)
        sph.compute_eos(gpu_ctx, d)
        sph.compute_iad_divv_curlv(gpu_ctx, d)
        sph.compute_av_switches(gpu_ctx, d)
        gpu_ctx.set_deterministic(det)
        edit(d)
        sph.compute_momentum_energy(gpu_ctx, d, clean)
        out[det] = {f: d.f[f].cpu().numpy() for f in ME_FIELDS}
        out[det]["minDt"] = d.minDtCourant
    gpu_ctx.set_deterministic(False)
    return out[False], out[True]


def check_me(once, fixed):
    for f in ME_FIELDS:
        assert np.all(np.isfinite(fixed[f])), f
        err = np.max(np.abs(once[f] - fixed[f])) / field_scale(fixed, f)
        assert err <= 1e-12, f"{f}: {err:.3e}"
    assert once["minDt"] == pytest.approx(fixed["minDt"], rel=1e-12)


@pytest.mark.parametrize("size", [1e-300, 1e-312, 1e-318, 1e-322])
def test_viscosity_cleaning_with_subnormal_velocity_gradients(gpu_ctx, size):
    """Velocity gradients that decay into the subnormal range (a smooth pulse far from its centre): the
    cleaning term of such pairs is next to nothing and must not become infinite."""
    def edit(d):
        for k in ("dV11", "dV12", "dV13", "dV22", "dV23", "dV33"):
            t = d.f[k]
            half = t.shape[0] // 2
            t[:half] = t[:half].sign() * size
            d.f["dV11"][:half] = size
            d.f["dV22"][:half] = size
    check_me(*momentum_energy_both(gpu_ctx, edit, clean=True))


def test_atwood_weights_where_the_sum_of_densities_leaves_fp32(gpu_ctx):
    """Densities that FP32 holds with sums that it does not: the decision between the flat branches and
    the ramp is the FP64 one."""
    import torch

    def edit(d):
        g = torch.Generator(device="cuda:0")
        g.manual_seed(5)
        rho = torch.empty_like(d.f["kx"]).uniform_(1.3e38, 3.3e38, generator=g)
        d.f["kx"].copy_(rho * d.f["xm"] / d.f["m"])
    check_me(*momentum_energy_both(gpu_ctx, edit))


@pytest.mark.parametrize("clean", [False, True])
@pytest.mark.parametrize("scale", [1e-200, 1e-170, 1e170, 1e200])
def test_masses_near_the_ends_of_the_exponent_range(gpu_ctx, scale, clean):
    """Masses of 1e+-200 with prho and kx of a caller's own equation of state: products of two masses leave
    the exponent range, the accelerations do not."""
    def edit(d):
        d.f["m"].mul_(scale)
        d.f["kx"].div_(scale)
        d.f["prho"].div_(scale)
    check_me(*momentum_energy_both(gpu_ctx, edit, clean=clean))


@pytest.mark.parametrize("scale", [1e-19, 1e-20, 1e-21, 1e-22, 1e-24, 1e-30])
@pytest.mark.parametrize("n, periodic", [(600, True), (1728, True), (6000, True), (3000, False)])
def test_neighbours_where_squared_radii_are_subnormal_in_fp32(gpu_ctx, port, n, periodic, scale):
    """Lengths whose squares FP32 holds with a few bits or none: neighbour counts of small periodic boxes
    (pairs folded one by one) and of an open set against the oracle."""
    from sphexa_gb300 import workloads as W
    wl = W.random_cube(n, seed=120 + n, periodic=periodic)
    for k in ("x", "y", "z", "h"):
        wl.fields[k] = wl.fields[k] * scale
    wl.box = wl.box * scale
    wl.fields["m"] = wl.fields["m"] * scale ** 3
    gpu_ctx.set_deterministic(False)
    r = run_gpu(gpu_ctx, wl, "std", False)
    ref = port.sweep(wl, "std", False)
    np.testing.assert_array_equal(r["nc"], ref["nc"])


@pytest.mark.parametrize("scale", [1e-30, 1e-24, 1e22, 1e28])
def test_search_prunes_nodes_in_any_unit(gpu_ctx, scale):
    """Lengths whose squares leave FP32: nodes are pruned as in ordinary units, single candidates are not.
    Pairs tested then: with nodes of at most 256 particles (edge 6.4 spacings) the region of 9 spacings
    grows to 21.7 at most, 16.5 times as many pairs as the 620 per target of ordinary units; without
    pruning it would be every pair of the set, 97 times."""
    from sphexa_gb300 import workloads as W
    tested = []
    for f in (1.0, scale):
        wl = W.random_cube(60000, seed=140, periodic=False)
        for k in ("x", "y", "z", "h"):
            wl.fields[k] = wl.fields[k] * f
        wl.box = wl.box * f
        tested.append(run_gpu(gpu_ctx, wl, "std", False)["stats"]["candidates"])
    assert tested[1] <= 20 * tested[0], tested


@pytest.mark.parametrize("how", ["sweep", "passes"])
def test_undefined_std_results_show_where_the_order_fixed_form_has_them(gpu_ctx, how):
    """A pair of particles at one point has no distance, and what its densities reach is NaN in every output that
    takes them, du of receding neighbours included."""
    from sphexa_gb300 import sph, workloads as W
    wl = W.random_cube(1500, seed=201, periodic=False)
    rng = np.random.Generator(np.random.PCG64(202))
    for k in ("x", "y", "z"):
        wl.fields[k][1] = wl.fields[k][0]
    for k in ("vx", "vy", "vz"):
        wl.fields[k] = rng.normal(0.0, 0.2, wl.n).astype(np.float32).astype(np.float64)
    gpu_ctx.set_params(ng0=int(wl.params["ng0"]), ngmax=int(wl.params["ngmax"]), bucket=int(wl.params["bucket"]),
                       minDt=float(wl.params["minDt"]))
    out = {}
    for det in (True, False):
        gpu_ctx.set_deterministic(det)
        d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0")
        box = sph.Box(wl.box.copy(), wl.bc.copy())
        if how == "sweep":
            sph.sweep(gpu_ctx, d, box, "std")
        else:
            sph.Domain(gpu_ctx, box).sync(d)
            sph.find_neighbors_sfc(gpu_ctx, 0, wl.n, d)
            sph.compute_density(gpu_ctx, d)
            sph.compute_eos_hydro_std(gpu_ctx, d)
            sph.compute_iad(gpu_ctx, d)
            sph.compute_momentum_energy_std(gpu_ctx, d)
        out[det] = {f: np.isnan(d.f[f].cpu().numpy()) for f in ("rho", "c11", "ax", "ay", "az", "du")}
    gpu_ctx.set_deterministic(False)
    assert out[True]["du"].any()
    for f in out[True]:
        np.testing.assert_array_equal(out[False][f], out[True][f], f)
