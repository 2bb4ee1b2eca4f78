"""The work a user of this framework has it do, as timed cases.

Every case is one call (or one pair of calls) of a direct-SCF program: a Fock
build on host arrays through the reference's entry points, a build on device
arrays, an incremental mixed-precision build, a recorded build, a batch of
molecules, or a whole SCF job as the server runs it.  Molecules are the ones
the package generates (water clusters, n-alkanes, benzene, C60), displaced by
a seeded few hundredths of an Angstrom, as a geometry optimisation or a
dynamics run displaces them from step to step.

Densities come from a one-electron model Hamiltonian (kinetic energy, bare
nuclei and a neutralising Gaussian electron cloud on every atom), whose
occupied orbitals have the decay and the block sizes of converged ones; an
incremental build takes the difference of two such densities.  These and the
64-bit results of `exact` are plain torch (McMurchie-Davidson integrals over
the shells' exponents and coefficients) and share no integral code with the
package.
"""
import itertools
import math

import numpy as np
import torch

from hfcode_b200 import basis, fock, molecules, scf

THR = 1e-10         # integral threshold of a converging SCF
DELTA_FACTOR = 0.1  # non-diagonal threshold of an incremental build, relative to THR
CUTOFF = 1e-7       # FP32 below this bound in the incremental builds
SERVED_SCRATCH = 256 << 20  # scratch of one job of the server
BATCH = [("alkane", 4), ("alkane", 8), ("alkane", 12), ("alkane", 16),
         ("water", 3), ("water", 6), ("water", 9), ("water", 12)]


# ------------------------------------------------------------------ cases

def listed():
    return [
        # the smallest call: a minimal-basis water molecule through the
        # reference's two entry points on host arrays, as its program makes it
        {"name": "water_sto3g_host", "call": "host", "mol": "water", "n": 1, "basis": "STO-3G", "split": False, "shift": 0.02},
        # the same calls at the size of a small organic molecule
        {"name": "benzene_host", "call": "host", "mol": "benzene", "n": 1, "basis": "6-31G(d)", "split": False, "shift": 0.02},
        # a basis written with separate s and p shells, as most libraries write it
        {"name": "benzene_split_host", "call": "host", "mol": "benzene", "n": 1, "basis": "6-31G(d)", "split": True, "shift": 0.02},
        # one incremental cycle of a small served job: device arrays, mixed precision
        {"name": "water3_delta", "call": "delta", "mol": "water", "n": 3, "basis": "6-31G(d)", "split": False, "shift": 0.02},
        # a host SCF driver that replays its recorded build each cycle
        {"name": "c8h18_graph", "call": "graph", "mol": "alkane", "n": 8, "basis": "6-31G(d)", "split": False, "shift": 0.02},
        # a Coulomb-only build of a medium chain
        {"name": "c16h34_j_host", "call": "host_j", "mol": "alkane", "n": 16, "basis": "6-31G(d)", "split": False, "shift": 0.02},
        # a full FP64 device build of a compact, medium system
        {"name": "water12_full", "call": "full", "mol": "water", "n": 12, "basis": "6-31G(d)", "split": False, "shift": 0.02},
        # eight molecules of the served range in one launch
        {"name": "batch8", "call": "batch", "mol": "mixed", "n": 8, "basis": "6-31G(d)", "split": False, "shift": 0.02},
        # a whole served job, from the handle to the converged density
        {"name": "water5_job", "call": "job", "mol": "water", "n": 5, "basis": "6-31G(d)", "split": False, "shift": 0.02},
        # the mixed form's own configuration: n-C20H42, incremental, cutoff 1e-7
        {"name": "c20h42_delta", "call": "delta", "mol": "alkane", "n": 20, "basis": "6-31G(d)", "split": False, "shift": 0.02},
        # the headline: C60, one full FP64 build on device arrays
        {"name": "c60_full", "call": "full", "mol": "c60", "n": 1, "basis": "6-31G(d)", "split": False, "shift": 0.02},
        # the later cycles of the same SCF in the mixed form
        {"name": "c60_delta", "call": "delta", "mol": "c60", "n": 1, "basis": "6-31G(d)", "split": False, "shift": 0.02},
    ]


def draw(rng):
    """Another call on another molecule of the same ranges."""
    call = rng.choice(["host", "host_j", "full", "delta", "graph", "job"])
    mol = rng.choice(["water", "alkane"])
    most = {"water": 8 if call == "job" else 20, "alkane": 10 if call == "job" else 30}[mol]
    n = min(most, int(math.exp(rng.uniform(0.0, math.log(most + 1.0)))))
    name = rng.choice(["6-31G(d)", "6-31G(d)", "6-31G(d)", "STO-3G"])
    split = call != "job" and rng.random() < 0.25
    if name == "STO-3G" and rng.random() < 0.2 and call != "job":
        mol, n = "c60", 1
    return {"call": call, "mol": mol, "n": n, "basis": name, "split": split,
            "shift": round(rng.uniform(0.01, 0.04), 4)}


# ------------------------------------------------------------- molecules

def ideal(mol, n):
    if mol == "water":
        return molecules.water() if n == 1 else molecules.water_cluster(n, np.random.default_rng(20261203 + n))
    if mol == "alkane":
        return molecules.alkane(n)
    return {"benzene": molecules.benzene, "c60": molecules.c60}[mol]()


def system(mol, n, basis_name, split, shift, seed):
    """(molecule, element basis, shells) of one geometry, every coordinate
    displaced by a normal deviate of `shift` Angstrom."""
    m = ideal(mol, n)
    move = np.random.default_rng([seed, n]).normal(scale=shift, size=m.coords_ang.shape)
    m = basis.Molecule(list(m.labels), m.coords_ang + move)
    bas = basis.load_basis(basis_name)
    sh = basis.spread_basis(m, bas)
    return m, bas, basis.split_l_shells(sh) if split else sh


# ------------------------------------- plain Gaussian integrals, in 64 bits

def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def carts(l):
    return [(l - i, i - k, k) for i in range(l + 1) for k in range(i + 1)]


def hermites(l):
    return [(t, u, v) for t in range(l + 1) for u in range(l + 1 - t) for v in range(l + 1 - t - u)]


R3 = math.sqrt(3.0)
# real solid harmonics z2, xz, yz, xy, x2-y2 over xx, xy, xz, yy, yz, zz
HARMONICS = [[-0.5, 0, 0, -0.5, 0, 1], [0, 0, R3, 0, 0, 0], [0, 0, 0, 0, R3, 0], [0, R3, 0, 0, 0, 0],
             [R3 / 2, 0, 0, -R3 / 2, 0, 0]]


def shell_groups(sh):
    """The shells as pure s, p and d shells (an sp shell is two of them), in
    groups of equal angular momentum and primitive count."""
    found = {}
    for i in range(sh.nsh):
        k, ao, c = int(sh.nzet[i]), int(sh.aosh[i]), sh.djk[i]
        parts = {basis.SHELL_S: [(0, ao, c)], basis.SHELL_P: [(1, ao, c)], basis.SHELL_D: [(2, ao, c)],
                 basis.SHELL_L: [(0, ao, c), (1, ao + 1, c * sh.djkl[i])]}[int(sh.shtyp[i])]
        for l, first, coef in parts:
            found.setdefault((l, k), []).append((sh.xsh[i], sh.zeta[i][:k], coef[:k], first))
    t = lambda rows: torch.tensor(np.array(rows), dtype=torch.float64, device=device())
    out = []
    for (l, _), rows in sorted(found.items()):
        ao = torch.tensor([r[3] for r in rows], device=device())
        out.append({"l": l, "x": t([r[0] for r in rows]), "z": t([r[1] for r in rows]), "c": t([r[2] for r in rows]),
                    "ao": ao[:, None] + torch.arange(2 * l + 1, device=device())})
    return out


def hermite_1d(la, lb, p, pa, pb, e0):
    """Expansion coefficients E[i, j][t] of the products x_A^i x_B^j."""
    E = {(0, 0): [e0]}
    for i, j in itertools.product(range(la + 1), range(lb + 1)):
        if i == j == 0:
            continue
        old, x = (E[i - 1, j], pa) if i else (E[i, j - 1], pb)
        get = lambda t: old[t] if 0 <= t < len(old) else torch.zeros_like(e0)
        E[i, j] = [get(t - 1) / (2 * p) + x * get(t) + (t + 1) * get(t + 1) for t in range(i + j + 1)]
    return E


def spherical(M, l, axis):
    if l < 2:
        return M
    h = torch.tensor(HARMONICS, dtype=torch.float64, device=M.device)
    return torch.movedim(torch.tensordot(M, h, dims=([axis], [1])), -1, axis)


def shell_pairs(g, k):
    """Every pair of a shell of group g with one of group k: exponent sums and
    centres [pair, primitive], Hermite coefficients [pair, primitive, functions,
    Hermite], and overlap and kinetic blocks."""
    na, nb, la, lb = len(g["x"]), len(k["x"]), g["l"], k["l"]
    a, b = g["z"][:, None, :, None], k["z"][None, :, None, :]
    w = (g["c"][:, None, :, None] * k["c"][None, :, None, :]).reshape(na * nb, -1)
    shape = (na, nb, g["z"].shape[1], k["z"].shape[1])
    A, B = g["x"][:, None, None, None, :], k["x"][None, :, None, None, :]
    flat = lambda v: v.expand(shape).reshape(na * nb, -1)
    p = flat(a + b)
    P = [flat((a * A[..., d] + b * B[..., d]) / (a + b)) for d in range(3)]
    E = [hermite_1d(la, lb + 2, p, P[d] - flat(A[..., d]), P[d] - flat(B[..., d]),
                    torch.exp(-flat(a * b / (a + b) * (A[..., d] - B[..., d]) ** 2))) for d in range(3)]
    zb = flat(b)
    zero = torch.zeros_like(p)
    kin = lambda d, i, j: (-2 * zb * zb * E[d][i, j + 2][0] + zb * (2 * j + 1) * E[d][i, j][0]
                           - (0.5 * j * (j - 1) * E[d][i, j - 2][0] if j > 1 else 0.0))
    H, S, T = [], [], []
    root = (math.pi / p) ** 1.5 * w
    for ca, cb in itertools.product(carts(la), carts(lb)):
        e = [E[d][ca[d], cb[d]] for d in range(3)]
        H.append(torch.stack([w * e[0][t] * e[1][u] * e[2][v]
                              if t < len(e[0]) and u < len(e[1]) and v < len(e[2]) else zero
                              for t, u, v in hermites(la + lb)], dim=-1))
        S.append((root * e[0][0] * e[1][0] * e[2][0]).sum(1))
        q = [kin(d, ca[d], cb[d]) for d in range(3)]
        T.append((root * (q[0] * e[1][0] * e[2][0] + e[0][0] * q[1] * e[2][0] + e[0][0] * e[1][0] * q[2])).sum(1))

    def functions(M, rest):  # [pair, (cart a, cart b), rest] to [pair, functions, rest]
        M = M.reshape((na * nb, len(carts(la)), len(carts(lb))) + rest)
        M = spherical(spherical(M, la, 1), lb, 2)
        return M.reshape((na * nb, (2 * la + 1) * (2 * lb + 1)) + rest)

    H = functions(torch.stack(H, dim=1).reshape(na * nb, -1, p.shape[1] * len(hermites(la + lb))),
                  (p.shape[1] * len(hermites(la + lb)),))
    H = H.reshape(na * nb, H.shape[1], p.shape[1], -1).permute(0, 2, 1, 3).contiguous()
    ia = g["ao"][:, None, :, None].expand(na, nb, -1, k["ao"].shape[1]).reshape(na * nb, -1)
    ib = k["ao"][None, :, None, :].expand(na, nb, g["ao"].shape[1], -1).reshape(na * nb, -1)
    return {"l": la + lb, "p": p, "P": P, "H": H, "S": functions(torch.stack(S, dim=1), ()),
            "T": functions(torch.stack(T, dim=1), ()), "ia": ia, "ib": ib}


def boys(M, T):
    """F_0 .. F_M: the ascending series of F_M and downward recursion below
    T = 36, upward recursion from the error function above."""
    small = torch.clamp(T, max=36.0)
    term = torch.full_like(T, 1.0 / (2 * M + 1))
    total = term.clone()
    for i in range(1, 130):
        term = term * (2 * small / (2 * M + 2 * i + 1))
        total = total + term
    ex = torch.exp(-small)
    low = [None] * M + [ex * total]
    for m in range(M - 1, -1, -1):
        low[m] = (2 * small * low[m + 1] + ex) / (2 * m + 1)
    big = torch.clamp(T, min=36.0)
    exb = torch.exp(-big)
    high = [0.5 * torch.sqrt(math.pi / big) * torch.erf(torch.sqrt(big))]
    for m in range(M):
        high.append(((2 * m + 1) * high[m] - exb) / (2 * big))
    return [torch.where(T < 36.0, x, y) for x, y in zip(low, high)]


def hermite_coulomb(L, alpha, X):
    """R[t, u, v] of the Hermite Coulomb integrals, t + u + v <= L."""
    F = boys(L, alpha * (X[0] ** 2 + X[1] ** 2 + X[2] ** 2))
    level = {(0, 0, 0): [(-2 * alpha) ** n * F[n] for n in range(L + 1)]}
    for t, u, v in sorted(hermites(L), key=sum):
        if t + u + v == 0:
            continue
        d = 0 if t else 1 if u else 2
        one = list((t, u, v)); one[d] -= 1
        two = list(one); two[d] -= 1
        count = L + 1 - (t + u + v)
        level[t, u, v] = [X[d] * level[tuple(one)][n + 1]
                          + (one[d] * level[tuple(two)][n + 1] if one[d] else 0.0) for n in range(count)]
    return {k: v[0] for k, v in level.items()}


def put(M, pair, block):
    M[pair["ia"], pair["ib"]] = block
    M[pair["ib"], pair["ia"]] = block


def all_pairs(sh):
    g = shell_groups(sh)
    return [shell_pairs(g[i], g[j]) for i in range(len(g)) for j in range(i + 1)]


def one_electron(mol, sh, pairs, clouds):
    """S, T and the potential of the nuclei; with `clouds` (a factor per atom on
    the exponents), also that of a neutralising Gaussian electron cloud on every
    atom, a tight core and a valence part: the potential of neutral atoms."""
    S, T, V = (torch.zeros(sh.nb, sh.nb, dtype=torch.float64, device=device()) for _ in range(3))
    charges = []  # (position, charge, exponent of the Gaussian or None)
    for i, (x, z) in enumerate(zip(mol.coords, mol.charges)):
        charges.append((x, -z, None))
        if clouds is not None:
            core = 2.0 if z > 2 else 0.0
            charges.append((x, z - core, (0.45 if z > 2 else 0.6) * clouds[i]))
            if core:
                charges.append((x, core, 0.6 * z * z * clouds[i]))
    for pr in pairs:
        put(S, pr, pr["S"])
        put(T, pr, pr["T"])
        acc = torch.zeros_like(pr["S"])
        hs = hermites(pr["l"])
        step = max(1, (1 << 20) // pr["p"].numel())
        for at in range(0, len(charges), step):  # a chunk of the charges at a time
            part = charges[at:at + step]
            q = torch.tensor([c[1] for c in part], dtype=torch.float64, device=device())[:, None, None]
            eta = torch.tensor([c[2] or 0.0 for c in part], dtype=torch.float64, device=device())[:, None, None]
            xyz = torch.tensor(np.array([c[0] for c in part]), dtype=torch.float64, device=device())
            f = torch.where(eta > 0, eta / (pr["p"] + eta), torch.ones_like(eta))
            R = hermite_coulomb(pr["l"], pr["p"] * f, [pr["P"][d] - xyz[:, d, None, None] for d in range(3)])
            w = 2 * math.pi / pr["p"] * torch.sqrt(f) * q
            W = torch.stack([(w * R[h]).sum(0) for h in hs], dim=-1)
            acc = acc + torch.einsum("kqfh,kqh->kf", pr["H"], W)
        put(V, pr, acc)
    return S, T, V


def repulsion_tensor(sh, pairs):
    """(ij|kl) over all functions as an nb^2 x nb^2 matrix."""
    nb = sh.nb
    G = torch.zeros(nb * nb, nb * nb, dtype=torch.float64, device=device())
    for x, bra in enumerate(pairs):
        for ket in pairs[:x + 1]:
            hb, hk = hermites(bra["l"]), hermites(ket["l"])
            sign = torch.tensor([(-1.0) ** sum(h) for h in hk], dtype=torch.float64, device=device())
            nk, qk = ket["p"].shape
            q = ket["p"].reshape(-1)[None, :]
            step = max(1, (1 << 19) // (bra["p"].shape[1] * q.numel()))
            for at in range(0, len(bra["p"]), step):
                sl = slice(at, at + step)
                p = bra["p"][sl].reshape(-1)[:, None]
                X = [bra["P"][d][sl].reshape(-1)[:, None] - ket["P"][d].reshape(-1)[None, :] for d in range(3)]
                R = hermite_coulomb(bra["l"] + ket["l"], p * q / (p + q), X)
                pref = 2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
                block = 0.0
                for i, h in enumerate(hb):
                    M = torch.stack([R[h[0] + k[0], h[1] + k[1], h[2] + k[2]] for k in hk]) * sign[:, None, None] * pref
                    Y = torch.einsum("hpkq,kqch->pkc", M.reshape(len(hk), -1, nk, qk), ket["H"])
                    E = bra["H"][sl][..., i]
                    block = block + torch.einsum("bpa,bpkc->bakc", E, Y.reshape(E.shape[0], E.shape[1], nk, -1))
                rows = [(bra["ia"][sl] * nb + bra["ib"][sl]).reshape(-1), (bra["ib"][sl] * nb + bra["ia"][sl]).reshape(-1)]
                cols = [(ket["ia"] * nb + ket["ib"]).reshape(-1), (ket["ib"] * nb + ket["ia"]).reshape(-1)]
                block = block.reshape(len(rows[0]), len(cols[0]))
                for r, c in itertools.product(rows, cols):
                    G[r[:, None], c[None, :]] = block
                    G[c[:, None], r[None, :]] = block.T
    return G


def coulomb(G, P):
    return (G @ P.reshape(-1)).reshape(P.shape)


def exchange(G, P):
    n = P.shape[0]
    return torch.einsum("ijkl,jl->ik", G.reshape(n, n, n, n), P)


# --------------------------------------------------------------- densities

def inverse_root(S):
    e, U = torch.linalg.eigh(S)
    return (U / torch.sqrt(e)) @ U.T


def occupied(H, X, nocc):
    _, C = torch.linalg.eigh(X @ H @ X)
    C = (X @ C)[:, :nocc]
    P = 2.0 * C @ C.T
    return 0.5 * (P + P.T)


def densities(mol, sh, seed):
    """The core Hamiltonian, a density and the change an SCF cycle makes to it."""
    pairs = all_pairs(sh)
    S, T, V = one_electron(mol, sh, pairs, clouds=None)
    _, _, W = one_electron(mol, sh, pairs, clouds=np.ones(mol.natom))
    X = inverse_root(S)
    P = occupied(T + W, X, mol.nocc)
    # the change: what a small breathing of every atom's cloud does to the density
    scale = 1.0 + np.random.default_rng([seed, 1]).normal(scale=0.005, size=mol.natom)
    _, _, W2 = one_electron(mol, sh, pairs, clouds=scale)
    dP = occupied(T + W2, X, mol.nocc) - P
    return T + V, P, dP


# ---------------------------------------------------------- prepare and run

def molecule_state(call, mol, n, basis_name, split, shift, seed):
    m, bas, sh = system(mol, n, basis_name, split, shift, seed)
    H, P, dP = densities(m, sh, seed)
    fb = fock.FockBuilder(sh, scratch_budget=SERVED_SCRATCH if call == "batch" else None)
    f = np.zeros((sh.nb, sh.nb))
    p = P.cpu().numpy()
    fb.fock_build_initial_diag(f, p, THR)  # cycle 1: leaves the screening tables on the handle
    return {"sh": sh, "fb": fb, "H": H, "P": P, "dP": dP, "F": torch.empty_like(H),
            "h": H.cpu().numpy(), "p": p}


def prepare(case, seed):
    call = case["call"]
    if call == "job":
        m, bas, sh = system(case["mol"], case["n"], case["basis"], case["split"], case["shift"], seed)
        return {"call": call, "mol": m, "sh": sh, "p0": basis.density_superposition(m, bas, sh.nb)}
    if call == "batch":
        parts = [molecule_state(call, mol, n, case["basis"], case["split"], case["shift"], seed + 1000 * k)
                 for k, (mol, n) in enumerate(BATCH)]
        torch.cuda.synchronize()
        for s in parts:
            s["fb"].graph_capture(s["F"].data_ptr(), s["P"].data_ptr(), THR, THR, 0.0)
        return {"call": call, "parts": parts, "batch": fock.Batch([s["fb"] for s in parts]),
                "stream": torch.cuda.Stream()}
    s = molecule_state(call, case["mol"], case["n"], case["basis"], case["split"], case["shift"], seed)
    s["call"] = call
    s["stream"] = torch.cuda.ExternalStream(s["fb"].stream())
    if call == "graph":  # the recording an SCF driver makes in its second cycle
        s["fb"].fock_build_graph(s["h"].copy(), s["p"], THR, THR)
    torch.cuda.synchronize()
    return s


def run(state):
    call = state["call"]
    if call == "job":
        fb = fock.FockBuilder(state["sh"], scratch_budget=SERVED_SCRATCH)
        r = scf.device_hartreefock(state["mol"], state["sh"], fb, p_guess=state["p0"], maxiter=60, conv=1e-6,
                                   conve=1e-8, fp32_cutoff=CUTOFF)
        fb.close()
        return {"energy": r.energy, "P": r.P, "F": r.F, "eigs": r.eigs}
    if call == "batch":
        with torch.cuda.stream(state["stream"]):
            for s in state["parts"]:
                s["F"].copy_(s["H"])
        state["batch"].launch(state["stream"].cuda_stream)
        return [s["F"] for s in state["parts"]]
    fb = state["fb"]
    if call in ("host", "host_j"):
        f = state["h"].copy()
        fb.fock_build_diag(f, state["p"], THR)
        if call == "host":
            fb.fock_build_non_diag(f, state["p"], THR)
        else:
            fb.fock_build_non_diag_j_only(f, state["p"], THR)
        return f
    if call == "graph":
        f = state["h"].copy()
        fb.fock_build_graph(f, state["p"], THR, THR)
        return f
    F = state["F"]
    with torch.cuda.stream(state["stream"]):  # the builder's own stream
        if call == "full":
            F.copy_(state["H"])
            fb.fock_build_device(F.data_ptr(), state["P"].data_ptr(), THR, THR)
        else:
            F.zero_()
            fb.fock_build_device(F.data_ptr(), state["dP"].data_ptr(), THR, THR * DELTA_FACTOR, CUTOFF)
    return F


# ------------------------------------------------------------ exact results

def reference_scf(mol, sh, pairs, G):
    """RHF to well below the job's own convergence, with DIIS."""
    S, T, V = one_electron(mol, sh, pairs, clouds=None)
    _, _, W = one_electron(mol, sh, pairs, clouds=np.ones(mol.natom))
    H, X = T + V, inverse_root(S)
    P = occupied(T + W, X, mol.nocc)
    Fs, Rs = [], []
    for _ in range(60):
        F = H + coulomb(G, P) - 0.5 * exchange(G, P)
        R = X @ (F @ P @ S - S @ P @ F) @ X
        Fs, Rs = (Fs + [F])[-8:], (Rs + [R])[-8:]
        if R.abs().max() < 1e-10:
            break
        n = len(Fs)
        B = torch.zeros(n + 1, n + 1, dtype=torch.float64, device=device())
        B[:n, :n] = torch.stack([torch.stack([(a * b).sum() for b in Rs]) for a in Rs])
        B[n, :n] = B[:n, n] = -1.0
        rhs = torch.zeros(n + 1, dtype=torch.float64, device=device())
        rhs[n] = -1.0
        c = torch.linalg.lstsq(B.cpu(), rhs.cpu()[:, None]).solution[:n, 0]
        P = occupied(sum(float(x) * f for x, f in zip(c, Fs)), X, mol.nocc)
    x, z = mol.coords, mol.charges
    enuc = sum(z[i] * z[j] / float(np.linalg.norm(x[i] - x[j])) for i in range(len(z)) for j in range(i))
    return {"energy": 0.5 * float((P * (H + F)).sum()) + float(enuc), "P": P, "F": F,
            "eigs": torch.linalg.eigvalsh(X @ F @ X)}


def exact(case, seed):
    """All integrals kept, in 64 bits; only for molecules whose full tensor of
    repulsion integrals is quickly made."""
    call = case["call"]
    if call == "batch":
        return None
    mol, _, sh = system(case["mol"], case["n"], case["basis"], case["split"], case["shift"], seed)
    if sh.nb > 110:
        return None
    pairs = all_pairs(sh)
    G = repulsion_tensor(sh, pairs)
    if call == "job":
        return reference_scf(mol, sh, pairs, G)
    H, P, dP = densities(mol, sh, seed)
    if call == "delta":
        return coulomb(G, dP) - 0.5 * exchange(G, dP)
    if call == "host_j":  # the pairs' own quartets (ab|ab) keep their exchange
        nf = {basis.SHELL_S: 1, basis.SHELL_P: 3, basis.SHELL_D: 5, basis.SHELL_L: 4}
        of = torch.zeros(sh.nb, dtype=torch.int64, device=device())
        for i in range(sh.nsh):
            of[int(sh.aosh[i]):int(sh.aosh[i]) + nf[int(sh.shtyp[i])]] = i
        pair = (torch.maximum(of[:, None], of) * sh.nsh + torch.minimum(of[:, None], of)).reshape(-1)
        own = torch.where(pair[:, None] == pair[None, :], G, torch.zeros((), dtype=torch.float64, device=device()))
        return H + coulomb(G, P) - 0.5 * exchange(own, P)
    return H + coulomb(G, P) - 0.5 * exchange(G, P)


# --------------------------------------------------------------------- work

def build_work(mol, n, basis_name, split, thr):
    """Bytes and operations of one build: F read and written and P read once,
    the pairs' data read once; for every shell quartet whose bound (from the
    overlap of the two pairs' most diffuse primitives) reaches the threshold,
    60 operations per primitive quartet (the Boys function and the set-up) and
    14 per function quartet (six multiply-adds into J and K, and its
    accumulation)."""
    _, _, sh = system(mol, n, basis_name, split, 0.0, 0)
    z = np.array([sh.zeta[i][:sh.nzet[i]].min() for i in range(sh.nsh)])
    nf = np.array([{basis.SHELL_S: 1, basis.SHELL_P: 3, basis.SHELL_D: 5, basis.SHELL_L: 4}[int(t)] for t in sh.shtyp])
    i, j = np.tril_indices(sh.nsh)
    r2 = ((sh.xsh[i] - sh.xsh[j]) ** 2).sum(1)
    bound = np.exp(-z[i] * z[j] / (z[i] + z[j]) * r2)
    order = np.argsort(-bound)
    bound, functions, prims = bound[order], (nf[i] * nf[j])[order], (sh.nzet[i] * sh.nzet[j])[order]
    reach = np.searchsorted(-bound, -thr / np.maximum(bound, 1e-300), side="right")
    cf, cp = np.concatenate([[0], np.cumsum(functions)]), np.concatenate([[0], np.cumsum(prims)])
    quartets, primitives = 0.5 * float((functions * cf[reach]).sum()), 0.5 * float((prims * cp[reach]).sum())
    kept = int((bound > 1e-11).sum())
    return {"bytes": 24.0 * sh.nb ** 2 + 64.0 * float(prims[:kept].sum()), "flops": 60.0 * primitives + 14.0 * quartets}


def work(case):
    call = case["call"]
    if call == "batch":
        parts = [build_work(mol, n, case["basis"], case["split"], THR) for mol, n in BATCH]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    w = build_work(case["mol"], case["n"], case["basis"], case["split"], THR * (DELTA_FACTOR if call == "delta" else 1))
    if call == "job":  # about a dozen cycles, and each one's dense algebra (some 35 products of nb x nb)
        nb = math.sqrt(w["bytes"] / 24.0)
        w = {"bytes": 12 * w["bytes"], "flops": 12 * (w["flops"] + 35 * 2 * nb ** 3)}
    return w
