"""The FP64 pass variants chosen by size, list form or field values, against the CPU oracle at the sizes
and values where their branches change.  Bars as in test_gpu_parity.py: 1e-12 of the field's magnitude,
scaled by the conditioning of gradh for the fields downstream of it."""

import numpy as np
import pytest

from test_gpu_parity import field_scale, fp64_tol, run_gpu

pytestmark = pytest.mark.gpu

VE_FIELDS = ("rho", "p", "c", "xm", "kx", "gradh", "prho", "c11", "c12", "c13", "c22", "c23", "c33", "divv", "curlv",
             "alpha", "ax", "ay", "az", "du")


def check_fields(r, ref, variant, fields, what):
    for f in fields:
        err = np.max(np.abs(r[f] - ref[f])) / field_scale(ref, f)
        assert err <= fp64_tol(ref, f, variant), f"{what} {f}: {err:.3e}"


@pytest.mark.parametrize("spread", [0.02, 0.2, 1.0])
def test_atwood_branches_match_oracle(gpu_ctx, port, spread):
    """Masses spread by 10^(+-spread): pairs on the flat Atwood branches, on the ramp, and (spread 1) on
    the ramp with |ln xm_j - ln xm_i| s beyond the exponential table's range."""
    from sphexa_gb300 import workloads as W
    wl = W.fourier(14, seed=71, rho_seed=72, v_seed=73)
    rng = np.random.Generator(np.random.PCG64(74))
    wl.fields["m"] = (wl.fields["m"] * 10.0 ** rng.uniform(-spread, spread, wl.n)).astype(np.float32).astype(np.float64)
    gpu_ctx.set_deterministic(False)
    r = run_gpu(gpu_ctx, wl, "ve", False)
    ref = port.sweep(wl, "ve", False)
    check_fields(r, ref, "ve", VE_FIELDS, f"spread {spread}")


@pytest.mark.parametrize("name", ["fourier", "sphere", "few_neighbours"])
def test_avclean_once_matches_oracle(gpu_ctx, port, name):
    """Viscosity cleaning, one evaluation per mutual pair: lattice and clustered sets, and a set whose
    lists are short (wide eta_crit)."""
    from sphexa_gb300 import workloads as W
    wl = {"fourier": lambda: W.fourier(13, seed=75, rho_seed=76, v_seed=77),
          "sphere": lambda: W.sphere(4001, seed=78),
          "few_neighbours": lambda: W.random_cube(1500, seed=79)}[name]()
    rng = np.random.Generator(np.random.PCG64(80))
    for k in ("vx", "vy", "vz"):
        wl.fields[k] = rng.normal(0.0, 0.2, wl.n).astype(np.float32).astype(np.float64)
    if name == "few_neighbours":
        wl.params["ng0"], wl.params["ngmax"] = 40, 90
        wl.fields["h"] = (wl.fields["h"] * 0.7).astype(np.float32).astype(np.float64)
    gpu_ctx.set_deterministic(False)
    r = run_gpu(gpu_ctx, wl, "ve", True)
    ref = port.sweep(wl, "ve", True)
    np.testing.assert_array_equal(r["nc"], ref["nc"])
    check_fields(r, ref, "ve", VE_FIELDS, name)
    assert r["minDt"] == pytest.approx(float(ref["minDtCourant"]), rel=1e-12)


@pytest.mark.parametrize("n", [33, 640, 1331])
@pytest.mark.parametrize("masses", ["equal", "spread"])
def test_std_once_matches_oracle(gpu_ctx, port, n, masses):
    """The std chain with one evaluation per mutual pair, in a sweep (cached geometry) and pass by pass
    (geometry formed in every pass): partly filled warps and blocks, equal and unequal masses."""
    from sphexa_gb300 import sph, workloads as W
    wl = W.random_cube(n, seed=81 + n, periodic=n > 600)
    rng = np.random.Generator(np.random.PCG64(82))
    m = np.full(n, 1.0 / n) if masses == "equal" else 10.0 ** rng.uniform(-0.5, 0.5, n) / n
    wl.fields["m"] = m.astype(np.float32).astype(np.float64)
    fields = ("rho", "p", "c", "c11", "c12", "c13", "c22", "c23", "c33", "ax", "ay", "az", "du")
    gpu_ctx.set_deterministic(False)
    r = run_gpu(gpu_ctx, wl, "std", False)
    ref = port.sweep(wl, "std", False)
    check_fields(r, ref, "std", fields, f"sweep {n} {masses}")
    assert r["minDt"] == pytest.approx(float(ref["minDtCourant"]), rel=1e-12)
    d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0")
    box = sph.Box(wl.box.copy(), wl.bc.copy())
    sph.Domain(gpu_ctx, box).sync(d)
    sph.find_neighbors_sfc(gpu_ctx, 0, wl.n, d)
    sph.compute_density(gpu_ctx, d)
    sph.compute_eos_hydro_std(gpu_ctx, d)
    sph.compute_iad(gpu_ctx, d)
    sph.compute_momentum_energy_std(gpu_ctx, d)
    check_fields({f: d.f[f].cpu().numpy() for f in fields}, ref, "std", fields, f"passes {n} {masses}")
    assert d.minDtCourant == pytest.approx(float(ref["minDtCourant"]), rel=1e-12)


@pytest.mark.parametrize("n", [257, 1728, 6000])
@pytest.mark.parametrize("edges", [(1.0, 1.0, 1.0), (1.0, 0.3, 0.3)])
def test_search_folds_small_periodic_boxes(gpu_ctx, port, n, edges):
    """Search boxes that reach half a periodic box (pairs folded one by one) and just stay below (offsets
    wrapped against the group's origin): neighbour sets against the oracle, cubic and flat boxes."""
    from sphexa_gb300 import workloads as W
    from test_gpu_parity import flat_sets
    h = 0.5 * (3.0 / (4.0 * np.pi) * 100 * np.prod(edges) / n) ** (1.0 / 3.0)
    wl = W.random_cube(n, seed=90 + n, periodic=True, h=h)
    for k, f in enumerate(("x", "y", "z")):
        wl.fields[f] = wl.fields[f] * edges[k]
        wl.box[2 * k + 1] = edges[k]
    r = run_gpu(gpu_ctx, wl, "std", False)
    ref = port.sweep(wl, "std", False)
    ng = int(wl.params["ngmax"])
    np.testing.assert_array_equal(r["keys"], ref["keys"])
    np.testing.assert_array_equal(r["nc"], ref["nc"])
    np.testing.assert_array_equal(flat_sets(r["nbr"], r["nc"], ng), flat_sets(ref["nbr"], ref["nc"], ng))


@pytest.mark.parametrize("scale", [1.0, 1e-18, 1e20])
@pytest.mark.parametrize("periodic", [True, False])
def test_mutual_pairs_of_varied_h(gpu_ctx, port, scale, periodic):
    """Lists and owned lists of equal, nearly equal and varied h, in units whose squared radii FP32 holds,
    flushes and overflows (every slot of a partial block is then inside the FP32 margin): the pair-once
    passes against the order-fixed ones, and the neighbour counts against the oracle."""
    from sphexa_gb300 import sph, workloads as W
    wl = W.random_cube(3000, seed=95, periodic=periodic)
    h0 = wl.fields["h"].mean()
    pick = np.arange(wl.n) % 4
    wl.fields["h"] = np.where(pick == 0, h0, np.where(pick == 1, h0 * (1 + 2.0 ** -45), np.where(
        pick == 2, h0 * (1 + 2.0 ** -25), wl.fields["h"])))
    for k in ("x", "y", "z", "h"):
        wl.fields[k] = wl.fields[k] * scale
    wl.box = wl.box * scale
    wl.fields["m"] = wl.fields["m"] * scale ** 3
    out = {}
    for det in (True, False):
        gpu_ctx.set_deterministic(det)
        out[det] = run_gpu(gpu_ctx, wl, "ve", False)
    gpu_ctx.set_deterministic(False)
    np.testing.assert_array_equal(out[False]["nc"], port.sweep(wl, "ve", False)["nc"])
    for f in ("xm", "kx", "gradh", "rho", "divv", "c11"):
        err = np.max(np.abs(out[False][f] - out[True][f])) / field_scale(out[True], f)
        assert err <= fp64_tol(out[True], f, "ve"), f"{f}: {err:.3e}"


@pytest.mark.parametrize("moved", ["nothing", "x", "vy", "h", "one_v"])
@pytest.mark.parametrize("variant", ["ve", "ve_clean", "std"])
def test_inputs_changed_between_passes(gpu_ctx, moved, variant):
    """Called one by one the passes share the pair geometry stored by the first as long as x, v and h are
    bit for bit what it saw; a change between passes (one component of one particle included) shows in the
    later passes as it does in the order-fixed form."""
    from sphexa_gb300 import sph, workloads as W
    wl = W.fourier(13, seed=96, rho_seed=97, v_seed=98)
    clean = variant == "ve_clean"
    fields = ("rho", "c11", "ax", "ay", "az", "du") + (() if variant == "std" else ("kx", "gradh", "divv", "alpha"))
    out = {}
    for det in (True, False):
        gpu_ctx.set_deterministic(det)
        d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0", av_clean=clean)
        box = sph.Box(wl.box.copy(), wl.bc.copy())
        sph.Domain(gpu_ctx, box).sync(d)
        sph.find_neighbors_sfc(gpu_ctx, 0, wl.n, d)
        (sph.compute_density if variant == "std" else sph.compute_xmass)(gpu_ctx, d)
        if moved == "one_v":
            d.f["vz"][wl.n // 2] += 0.5
        elif moved != "nothing":
            d.f[moved].mul_(1.0 + 1e-3)
        if variant == "std":
            sph.compute_eos_hydro_std(gpu_ctx, d)
            sph.compute_iad(gpu_ctx, d)
            sph.compute_momentum_energy_std(gpu_ctx, d)
        else:
            sph.compute_ve_def_gradh(gpu_ctx, d)
            sph.compute_eos(gpu_ctx, d)
            sph.compute_iad_divv_curlv(gpu_ctx, d)
            sph.compute_av_switches(gpu_ctx, d)
            sph.compute_momentum_energy(gpu_ctx, d, clean)
        out[det] = {f: d.f[f].cpu().numpy() for f in fields}
        out[det]["minDt"] = d.minDtCourant
    gpu_ctx.set_deterministic(False)
    check_fields(out[False], out[True], "std" if variant == "std" else "ve", fields, f"{variant} {moved}")
    assert out[False]["minDt"] == pytest.approx(out[True]["minDt"], rel=1e-12)


@pytest.mark.parametrize("n", [4096, 4097, 6001, 70001])
@pytest.mark.parametrize("spread", ["uniform", "cells", "cluster", "coincident"])
def test_sync_order_of_close_keys(gpu_ctx, n, spread):
    """The key sort by upper bits: sets without and with runs of keys that agree there (particles within
    a few grid cells of one another), one tight cluster (sorted over all bits) and equal keys (input
    order): order and keys against numpy's stable sort of the keys of an unsorted call."""
    import torch
    from sphexa_gb300 import _lib, sph, workloads as W
    wl = W.random_cube(n, seed=99, periodic=True)
    rng = np.random.Generator(np.random.PCG64(100))
    for k in ("x", "y", "z"):
        x = wl.fields[k]
        if spread == "cells":
            x = x[np.arange(n) // 5] + rng.uniform(0.0, 4e-6, n)
        elif spread == "cluster":
            x = 0.3 + rng.uniform(0.0, 1e-4, n)
        elif spread == "coincident":
            x = x[np.arange(n) // 7]
        wl.fields[k] = np.clip(x, 0.0, 1.0 - 1e-9)
    d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0")
    keys = torch.empty(n, dtype=torch.int64, device="cuda:0")
    box = sph.Box(wl.box.copy(), wl.bc.copy())
    b = box.to_c()
    assert gpu_ctx.lib.sphgb_sfc_keys_noalloc(d.x.data_ptr(), d.y.data_ptr(), d.z.data_ptr(), n, _lib.C.byref(b),
                                              keys.data_ptr(), None) == 0
    raw = keys.cpu().numpy().view(np.uint64)
    dom = sph.Domain(gpu_ctx, box)
    dom.sync(d)
    order = np.argsort(raw, kind="stable")
    np.testing.assert_array_equal(dom.order(n), order)
    np.testing.assert_array_equal(d.keys.cpu().numpy().view(np.uint64), raw[order])


@pytest.mark.parametrize("precision, bar", [("fp64", 1e-11), ("mixed", 1e-5)])
@pytest.mark.parametrize("du", [False, True])
@pytest.mark.parametrize("side", [9, 40])
def test_std_adjoint_over_owned_lists(side, du, precision, bar):
    """The std adjoint over owned lists (FP64: cut into 16 slices at 729 particles, 5 at 64,000; mixed:
    sums in 64-byte records, an odd count and a whole number of blocks) against the walk over the full
    lists.  Both add the same terms in different orders: about 150 terms a sum and four chained sums,
    each rounded to 1.1e-16 (6e-8) of the partial sum, so the bars leave a factor of a hundred (thirty)
    for cancellation between terms.  du: with and without a du seed (a kernel of its own each)."""
    import torch
    from sphexa_gb300 import autograd as AG, sph, workloads as W
    grads = {}
    for det in (False, True):
        wl = W.fourier(side, seed=3, rho_seed=31, v_seed=32, target_seed=33)
        ctx = sph.Context(0)
        d = sph.ParticlesData.from_workload(wl, precision, "cuda:0")
        box = sph.Box(wl.box.copy(), wl.bc.copy())
        sw = AG.FrozenStdSweep(ctx, d, box)
        sw.freeze()
        order = sph.Domain(ctx, box).order(wl.n)
        rho_t = torch.tensor(wl.fields["rho_target"][order], dtype=torch.float64, device="cuda:0")
        if det:
            ctx.set_deterministic(True)
        base = [t.clone().requires_grad_(True) for t in sw.inputs()]
        out = AG.StdSweepFunction.apply(sw, *base)
        loss = AG.loss_rho_a(*[o.to(torch.float64) for o in out[:4]], rho_t)
        if du:
            loss = loss + (out[4].to(torch.float64) ** 2).sum()
        loss.backward()
        grads[det] = [b.grad.detach().to(torch.float64) for b in base]
        ctx.close()
    for g1, g0 in zip(grads[False], grads[True]):
        assert float((g1 - g0).norm() / g0.norm()) <= bar


@pytest.mark.parametrize("n", [3000, 19456])
def test_small_set_densities_do_not_depend_on_the_order_of_atomics(gpu_ctx, n):
    """Sets in the most slices (up to 19,456 particles) keep the rounding errors of the xmass and gradh
    sums: hi + lo carries each sum to about 1e-32 of it in any order, so two sweeps round to the same
    bits."""
    from sphexa_gb300 import workloads as W
    wl = W.random_cube(n, seed=61, periodic=False)
    gpu_ctx.set_deterministic(False)
    a, b = run_gpu(gpu_ctx, wl, "ve", False), run_gpu(gpu_ctx, wl, "ve", False)
    for f in ("xm", "kx", "gradh"):
        assert np.array_equal(a[f], b[f]), f
