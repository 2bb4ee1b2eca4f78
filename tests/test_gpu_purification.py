"""The density step of the device SCF against an eigensolve.

After one cycle the job's density is the purified projector of X F X (no
extrapolation yet), so it must equal the one numpy's eigenvectors of the same
Fock matrix give.  Sizes cover both forms: the one-launch cluster kernel (one
tile; a ragged last tile; a multiple of the tile; its largest range) and the
product-per-step form beyond it.  Tolerance: the purification stops when
tr X - tr X^2 < 1e-11 nocc and then squares the rest twice, so the projector's
own error is below rounding; eigh and the dense products carry about
nb * eps * |P|, |P| <= 2.1, divided by the gap (>= 0.2 Eh of a spectrum of
about 30 Eh): 164 * 2.2e-16 * 2.1 * 150 = 1.2e-11.  1e-10 is asked for."""
import numpy as np
import pytest

from helpers import system


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["water", "wc1", "wc5", "benzene", "wc8", "alkane8", "alkane9"])
def test_purified_density_is_the_projector(name):
    from hfcode_b200 import onee
    from hfcode_b200.fock import DeviceSCFJob, FockBuilder
    mol, _, sh, p0 = system(name)
    S, T, V = onee.one_electron(mol, sh, gpu=True)
    fb = FockBuilder(sh)
    job = DeviceSCFJob(fb, mol.nocc, mol.nuclear_repulsion(), S, T + V, p0)
    r = job.run(maxiter=1)
    P, F, _ = job.get()
    job.close()
    fb.close()
    X = onee.s_minus_half(S)
    e, C = np.linalg.eigh(X @ F @ X)
    assert e[mol.nocc] - e[mol.nocc - 1] > 0.2
    C = (X @ C)[:, :mol.nocc]
    assert r["sp2_steps"] > 0
    assert np.max(np.abs(P - 2.0 * C @ C.T)) < 1e-10, sh.nb
