"""The form a recorded build gives its direct classes follows the work.

A recorded build's grids are capped, its candidates are not: water takes the
one launch over all direct classes, n-C20H42 and C60 in STO-3G (few classes,
long lists) a launch per class, the same kernels as with HFGPU_DIRECT=0.  The
replayed F equals the eager one: the same FP64 sums in another order, |F| up
to 60 with 1e6 terms an element, 1e-11."""
import numpy as np
import pytest

from hfcode_b200 import basis, molecules


def recorded(sh, p0, p, monkeypatch, direct):
    from hfcode_b200.fock import FockBuilder
    if direct is None:
        monkeypatch.delenv("HFGPU_DIRECT", raising=False)
    else:
        monkeypatch.setenv("HFGPU_DIRECT", direct)
    n = sh.nb
    fb = FockBuilder(sh)
    fb.fock_build_initial_diag(np.zeros((n, n)), p0, 1e-10)
    f, g = np.zeros((n, n)), np.zeros((n, n))
    fb.fock_build_diag(f, p, 1e-10)
    fb.fock_build_non_diag(f, p, 1e-10)
    before = fb.launch_count()
    fb.fock_build_graph(g, p, 1e-10, 1e-10)
    launches = fb.launch_count() - before
    fb.close()
    assert np.max(np.abs(f - g)) < 1e-11
    return launches


@pytest.mark.gpu
@pytest.mark.parametrize("name,small", [("water", True), ("c20h42", False), ("c60", False)])
def test_recorded_direct_form_follows_the_work(name, small, monkeypatch):
    mol = {"water": molecules.water, "c20h42": lambda: molecules.alkane(20), "c60": molecules.c60}[name]()
    bas = basis.load_basis("STO-3G")
    sh = basis.spread_basis(mol, bas)
    p0 = basis.density_superposition(mol, bas, sh.nb)
    d = np.random.default_rng(8).normal(size=p0.shape) * 0.01
    p = p0 + 0.5 * (d + d.T)
    own = recorded(sh, p0, p, monkeypatch, None)
    each = recorded(sh, p0, p, monkeypatch, "0")
    one = recorded(sh, p0, p, monkeypatch, "1000000000")
    assert one < each
    assert own == (one if small else each)
