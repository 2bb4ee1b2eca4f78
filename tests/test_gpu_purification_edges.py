"""Densities that purification cannot give: every orbital occupied, a matrix
that is a multiple of the identity, no gap at the occupation.

After one cycle the job's P is the density of X F X's nocc lowest eigenvectors.
Where the HOMO level is degenerate the choice among its vectors is free, so the
check is on what every choice gives: P S P = 2 P, tr P S = 2 nocc and
tr P F = 2 (sum of the nocc lowest eigenvalues).  Tolerance: eigensolves and
products of matrices of norm at most |F| (66 Eh for Ne, nb <= 180) carry
nb * eps * |F| = 2.6e-12 an element and at most nb of those in a trace: 1e-9."""
import numpy as np
import pytest

from hfcode_b200 import basis


def atoms(label, n, spacing):
    xyz = [[spacing * (i % 4), spacing * (i // 4 % 4), spacing * (i // 16)] for i in range(n)]
    mol, bas = basis.Molecule([label] * n, np.array(xyz, dtype=float)), basis.load_basis("STO-3G")
    sh = basis.spread_basis(mol, bas)
    return mol, sh, basis.density_superposition(mol, bas, sh.nb)


CASES = [("He", 1), ("He", 2), ("Ne", 1), ("O", 1), ("C", 1),          # one cluster launch
         ("He", 164), ("Ne", 36), ("O", 34)]                           # a product per step


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["job", "graph"])
@pytest.mark.parametrize("label,n", CASES)
def test_one_cycle_gives_a_density(label, n, form):
    from hfcode_b200 import onee
    from hfcode_b200.device_scf import DeviceSCF
    from hfcode_b200.fock import DeviceSCFJob, FockBuilder
    mol, sh, p0 = atoms(label, n, 8.0 if n > 2 else 3.0)
    S, T, V = onee.one_electron(mol, sh, gpu=True)
    fb = FockBuilder(sh)
    if form == "job":
        job = DeviceSCFJob(fb, mol.nocc, mol.nuclear_repulsion(), S, T + V, p0)
        job.run(maxiter=1)
        P, F, _ = job.get()
        job.close()
    else:
        r = DeviceSCF(mol, sh, fb, ints=(S, T, V)).run(p0, maxiter=1)
        P, F = r.P, r.F
    fb.close()
    X = onee.s_minus_half(S)
    e = np.linalg.eigvalsh(X @ F @ X)
    assert np.max(np.abs(P @ S @ P - 2.0 * P)) < 1e-9
    assert abs(np.sum(P * S) - 2.0 * mol.nocc) < 1e-9
    assert abs(np.sum(P * F) - 2.0 * np.sum(e[:mol.nocc])) < 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["job", "graph"])
@pytest.mark.parametrize("label,n", [("He", 1), ("He", 2), ("Ne", 1)])
def test_closed_shell_atoms_in_a_minimal_basis(label, n, form):
    """Converged energies against the oracle's SCF, 1e-8 Eh."""
    from hfcode_b200 import scf
    from hfcode_b200.device_scf import DeviceSCF
    from hfcode_b200.fock import FockBuilder
    from oracle import oscf
    mol, sh, p0 = atoms(label, n, 3.0)
    want = oscf.OracleSCF(mol.charges, mol.coords, mol.nocc, sh).run(p_guess=p0, conve=1e-10, conv=1e-7, maxiter=40)
    fb = FockBuilder(sh)
    kw = dict(conve=1e-10, conv=1e-7, maxiter=40)
    r = scf.device_hartreefock(mol, sh, fb, p_guess=p0, **kw) if form == "job" else \
        DeviceSCF(mol, sh, fb).run(p0, **kw)
    fb.close()
    assert want["converged"] and r.converged
    assert abs(r.energy - want["energy"]) < 1e-8
