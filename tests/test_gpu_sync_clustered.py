"""Syncs of tightly clustered sets, whose keys agree in more bits than the short sort looks at."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_clustered_sets_are_sorted_once(gpu_ctx):
    """The first sync of a tight cluster sorts by the upper bits (4 passes), finds runs that are too long, and
    sorts over all bits (8); the ones after it sort over all bits at once, whatever the set, for 31 syncs.
    Order and keys are numpy's stable sort of the keys throughout."""
    import torch
    from sphexa_gb300 import sph, workloads as W
    n = 70001
    ctx = sph.Context(0)
    rng = np.random.Generator(np.random.PCG64(151))
    sets = {}
    for name, width in (("cluster", 1e-4), ("uniform", 0.6)):
        wl = W.random_cube(n, seed=152, periodic=True)
        for k in ("x", "y", "z"):
            wl.fields[k] = 0.3 + width * rng.uniform(0.0, 1.0, n)
        sets[name] = wl

    def sync(name):
        wl = sets[name]
        d = sph.ParticlesData.from_workload(wl, "fp64", "cuda:0")
        box = sph.Box(wl.box.copy(), wl.bc.copy())
        b = box.to_c()
        raw = torch.empty(n, dtype=torch.int64, device="cuda:0")
        from sphexa_gb300 import _lib
        assert ctx.lib.sphgb_sfc_keys_noalloc(d.x.data_ptr(), d.y.data_ptr(), d.z.data_ptr(), n, _lib.C.byref(b),
                                              raw.data_ptr(), None) == 0
        raw = raw.cpu().numpy().view(np.uint64)
        before = ctx.launches()
        dom = sph.Domain(ctx, box)
        dom.sync(d)
        count = ctx.launches() - before
        order = np.argsort(raw, kind="stable")
        np.testing.assert_array_equal(dom.order(n), order)
        np.testing.assert_array_equal(d.keys.cpu().numpy().view(np.uint64), raw[order])
        return count

    first = sync("cluster")
    # 2 launches before the passes, 4 passes and the runs fewer
    assert [sync("cluster") for _ in range(31)] == [first - 7] * 31
    assert sync("cluster") == first
    long = [sync("uniform") for _ in range(31)]
    assert long == [long[0]] * 31
    assert sync("uniform") == long[0] - 3  # 4 of the 8 passes, and the runs
    ctx.close()
