"""The forms a build's lists can take give the same Fock matrix.

Which kernels run is chosen by the sizes of the lists: the direct classes in
one launch or one each, a staged chunk's roles on work units or one launch per
role, its scatter by one warp or one thread per quartet.  Each choice is forced
here at handle creation, together with a scratch budget that cuts the lists
into many chunks (the smallest is one tile of 128 quartets, so units straddle
chunk ends), for the full, the mixed, the Coulomb-only and the recorded build.

Tolerances: FP64 sums of the same terms in another order, |F| up to about 30
with 1e5 terms an element: 1e-11.  Mixed: both sides evaluate the quartets
below 1e-6 in FP32, each with up to 1e-6 relative error of at most 1e-6 times
the number of such quartets that meet in one element (below 1e4): 1e-8."""
import os

import numpy as np
import pytest

from helpers import perturbed_density, system
from oracle import pyoracle

FORMS = {
    "default": ({}, None),
    "direct_each": ({"HFGPU_DIRECT": "0"}, None),
    "roles_each": ({"HFGPU_MERGE_BLOCKS": "0", "HFGPU_WARP_SCATTER": "0"}, None),
    "all_units": ({"HFGPU_DIRECT": "100000000", "HFGPU_MERGE_BLOCKS": "100000000",
                   "HFGPU_WARP_SCATTER": "100000000"}, None),
    "unit_chunks": ({"HFGPU_MERGE_BLOCKS": "100000000"}, 4 << 20),
    "role_chunks": ({"HFGPU_MERGE_BLOCKS": "0", "HFGPU_WARP_SCATTER": "0"}, 4 << 20),
    "one_stream": ({"HFGPU_STREAMS": "1"}, 2 << 20),
}


def builds(sh, p0, p, env, budget):
    from hfcode_b200.fock import FockBuilder
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        fb = FockBuilder(sh, scratch_budget=budget)
    finally:
        for k, v in old.items():
            if v is None:
                os.environ.pop(k)
            else:
                os.environ[k] = v
    n = sh.nb
    fb.fock_build_initial_diag(np.zeros((n, n)), p0, 1e-10)
    out = {k: np.zeros((n, n)) for k in ("full", "mixed", "j", "graph")}
    fb.fock_build_non_diag(out["full"], p, 1e-10)
    passed = fb.class_stats()
    fb.fock_build_non_diag_mixed(out["mixed"], p, 1e-10, 1e-6)
    mixed = fb.class_stats()
    fb.fock_build_non_diag_j_only(out["j"], p, 1e-10)
    fb.fock_build_graph(out["graph"], p, 1e-10, 1e-10)
    diag = np.zeros((n, n))
    fb.fock_build_diag(diag, p, 1e-10)
    out["graph"] -= diag
    fb.close()
    return out, passed, mixed


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["water", "alkane2", "alkane2_mix", "wc3"])
def test_every_form_gives_the_same_matrix(name):
    _, _, sh, p0 = system(name)
    p = perturbed_density(p0, 4)
    orc = pyoracle.Oracle(sh)
    orc.fock_build_initial_diag(np.zeros((sh.nb, sh.nb)), p0, 1e-10)
    want = np.zeros((sh.nb, sh.nb))
    orc.fock_build_non_diag(want, p, 1e-10)
    first = None
    for form, (env, budget) in FORMS.items():
        out, passed, mixed = builds(sh, p0, p, env, budget)
        assert np.max(np.abs(out["full"] - want)) < 1e-10, form
        assert np.max(np.abs(out["graph"] - out["full"])) < 1e-11, form
        if first is None:
            first = out, passed, mixed
            continue
        for key, tol in (("full", 1e-11), ("j", 1e-11), ("mixed", 1e-8)):
            assert np.max(np.abs(out[key] - first[0][key])) < tol, (form, key)
        for key in ("pass", "scattered", "prim", "fp32"):  # whole numbers
            assert np.array_equal(passed[key], first[1][key]), (form, key)
        assert np.array_equal(mixed["pass"], first[2]["pass"]), form
        assert np.array_equal(mixed["prim"], first[2]["prim"]), form
