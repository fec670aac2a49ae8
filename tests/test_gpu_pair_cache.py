"""Memory of the FP64 pair-geometry cache: how much of the device it takes, and that it is given back."""

import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def free_memory(leave):
    """all but `leave` bytes of the device held by a tensor"""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda:0")
    try:
        yield
    finally:
        del fill
        torch.cuda.empty_cache()


def frozen(side, ctx):
    from sphexa_gb300 import autograd as AG, sph, workloads as W
    wl = W.fourier(side, seed=131, rho_seed=132, v_seed=133)
    d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0")
    sw = AG.FrozenVeSweep(ctx, d, sph.Box(wl.box.copy(), wl.bc.copy()), tape=False)
    sw.freeze()
    return wl, d, sw


def test_single_passes_take_an_eighth_of_the_free_memory():
    """27,000 particles, 120 MB of geometry, 400 MB free: a pass called by itself takes 50 MB of it (two of the
    five arrays, and the copy of its inputs)."""
    import torch
    from sphexa_gb300 import sph
    ctx = sph.Context(0)
    wl, d, sw = frozen(30, ctx)
    with free_memory(400 * MB):
        free = torch.cuda.mem_get_info()[0]
        sph.compute_xmass(ctx, d)
        used = free - torch.cuda.mem_get_info()[0]
    ctx.close()
    # an eighth, the copy of the inputs (1.5 MB), the sums (0.4 MB), and the allocator's 2 MB pages of each
    assert used <= free // 8 + 16 * MB, used


def test_cache_is_given_back_when_the_context_needs_the_space():
    """After a sweep that left 1.5 GB of geometry, with 160 MB free, the adjoint's 225 MB of state are found."""
    from sphexa_gb300 import sph
    ctx = sph.Context(0)
    wl, d, sw = frozen(70, ctx)
    vals = list(sw.inputs())
    rho, ax, ay, az, du = sw.forward(*vals)
    seeds = (2.0 * rho, 2.0 * ax, 2.0 * ay, 2.0 * az, None)
    with free_memory(160 * MB):
        g = [t.cpu().numpy() for t in sw.backward(*seeds)]
    assert all(np.all(np.isfinite(q)) for q in g)
    rho, ax, ay, az, du = sw.forward(*vals)  # and the passes go on
    again = [t.cpu().numpy() for t in sw.backward(*seeds)]
    for a, b in zip(g, again):
        assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(b))
    ctx.close()


def test_small_rises_of_the_pair_count_do_not_reallocate():
    """Twelve sweeps with h growing by 0.06 % each (2 % more pairs in all): one allocation."""
    from sphexa_gb300 import sph, workloads as W
    ctx = sph.Context(0)
    wl = W.fourier(30, seed=134, rho_seed=135, v_seed=136)
    d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0")
    box = sph.Box(wl.box.copy(), wl.bc.copy())
    pairs = []
    for step in range(12):
        sph.sweep(ctx, d, box, "ve")
        pairs.append(ctx.stats()["nc_sum"])
        d.f["h"].mul_(1.0006)
    assert 1.01 * pairs[0] < pairs[-1] < 1.03 * pairs[0], pairs
    cache = ctx.pair_cache()
    assert cache["arrays"] == 5 and cache["allocations"] == 1, cache
    ctx.close()


FIELDS = dict(ve=("xm", "kx", "gradh", "rho", "c11", "c23", "divv", "curlv", "alpha", "ax", "ay", "az", "du"),
              std=("rho", "c11", "c23", "ax", "ay", "az", "du"))


@pytest.mark.parametrize("arrays", [0, 2, 5])
@pytest.mark.parametrize("variant", ["ve", "ve_clean", "std"])
@pytest.mark.parametrize("how", ["sweep", "passes", "passes_moved"])
def test_every_form_of_the_cache_matches_the_order_fixed_passes(gpu_ctx, arrays, variant, how):
    """No cache, the two arrays of scalars, and all five, filled and read inside a sweep and by passes called
    one by one, with the same inputs and with velocities changed after the first pass."""
    from sphexa_gb300 import sph, workloads as W
    from test_gpu_parity import field_scale, fp64_tol
    wl = W.fourier(13, seed=141, rho_seed=142, v_seed=143)
    clean, chain = variant == "ve_clean", "std" if variant == "std" else "ve"
    gpu_ctx.set_params(ng0=int(wl.params["ng0"]), ngmax=int(wl.params["ngmax"]), bucket=int(wl.params["bucket"]),
                       minDt=float(wl.params["minDt"]))
    out = {}
    for det in (True, False):
        gpu_ctx.set_deterministic(det)
        gpu_ctx.set_pair_cache(0)
        gpu_ctx.set_pair_cache(arrays)
        d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0", av_clean=clean)
        box = sph.Box(wl.box.copy(), wl.bc.copy())
        if how == "sweep":
            sph.sweep(gpu_ctx, d, box, chain, clean)
        else:
            sph.Domain(gpu_ctx, box).sync(d)
            sph.find_neighbors_sfc(gpu_ctx, 0, wl.n, d)
            (sph.compute_density if chain == "std" else sph.compute_xmass)(gpu_ctx, d)
            if how == "passes_moved":
                d.f["vy"].mul_(1.01)
            if chain == "std":
                sph.compute_eos_hydro_std(gpu_ctx, d)
                sph.compute_iad(gpu_ctx, d)
                sph.compute_momentum_energy_std(gpu_ctx, d)
            else:
                sph.compute_ve_def_gradh(gpu_ctx, d)
                sph.compute_eos(gpu_ctx, d)
                sph.compute_iad_divv_curlv(gpu_ctx, d)
                sph.compute_av_switches(gpu_ctx, d)
                sph.compute_momentum_energy(gpu_ctx, d, clean)
        out[det] = {f: d.f[f].cpu().numpy() for f in FIELDS[chain]}
        out[det]["minDt"] = d.minDtCourant
        assert gpu_ctx.pair_cache()["arrays"] == (0 if det else arrays)
    gpu_ctx.set_deterministic(False)
    gpu_ctx.set_pair_cache(5)
    for f in FIELDS[chain]:
        err = np.max(np.abs(out[False][f] - out[True][f])) / field_scale(out[True], f)
        assert err <= fp64_tol(out[True], f, chain), f"{f}: {err:.3e}"
    assert out[False]["minDt"] == pytest.approx(out[True]["minDt"], rel=1e-12)


def test_cache_limits_are_checked(gpu_ctx):
    for bad in (-1, 1, 3, 6):
        with pytest.raises(Exception):
            gpu_ctx.set_pair_cache(bad)


def test_first_pass_repeated_alone_stops_storing():
    """xmass called again and again with no pass to read its geometry: the third call stores none, and the call
    after a pass that asked does."""
    from sphexa_gb300 import sph
    ctx = sph.Context(0)
    wl, d, sw = frozen(12, ctx)
    held = []
    for _ in range(4):
        sph.compute_xmass(ctx, d)
        held.append(ctx.pair_cache()["arrays"])
    assert held == [5, 5, 0, 0], held
    xm = d.f["xm"].cpu().numpy()
    sph.compute_ve_def_gradh(ctx, d)
    sph.compute_xmass(ctx, d)
    assert ctx.pair_cache()["arrays"] == 5
    np.testing.assert_allclose(d.f["xm"].cpu().numpy(), xm, rtol=1e-14)
    ctx.close()
