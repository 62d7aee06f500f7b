"""The density stage's shell slots in the tensor-core form: two of them while a
32-function tile touches few shells, one (with its own order of copies and waits)
above that, for GGA. Atoms of 16 functions each fill a tile in pairs, so the
shells of a tile are those of two atoms: 20 and 21 are the two sides of the
change at open shell, 24 and 25 at closed shell (pinned where the layout is
chosen, density_tc.cuh), 32 is the largest. Six atoms make three tiles, whose
slots are used again and again; all functions are in every group. Energy,
Kohn-Sham matrices and forces against the C restatement at the parity
tolerances, with and without the blocked basis."""
import numpy as np
import pytest

from lio_b200 import workloads as W

from . import helpers as H

pytestmark = pytest.mark.gpu

F_TOL = 1e-7  # Hartree / bohr, as the parity tests of the forces

# s, p and d shells of an atom: 16 functions in 10, 11, 12, 14 and 16 shells
A10, A11, A12, A14, A16 = (7, 3, 0), (10, 0, 1), (10, 2, 0), (13, 1, 0), (16, 0, 0)
CASES = [
    # (atoms of a pair, open shell, iexch)
    ((A10, A10), True, 9),
    ((A10, A11), True, 9),
    ((A16, A16), True, 9),
    ((A12, A12), False, 9),
    ((A11, A14), False, 9),
    ((A16, A16), False, 9),
    ((A16, A16), False, 3),
]


def molecule(pair, open_shell, iexch):
    mol = W.random_cluster({"H": 4, "C": 2}, 3.0, 17)
    shells = []
    for atom in range(1, 7):
        for l, n in enumerate(pair[(atom - 1) % 2]):
            shells += [(l, atom, 0.25 * 1.35 ** k * (1.0 + 0.1 * l)) for k in range(n)]
    M = 96
    q = W.random_orbitals(M, 5, np.random.default_rng(3))
    return H.shells_workload(mol, shells, W.pack_lower((1.0 if open_shell else 2.0) * q @ q.T, True), iexch, open_shell)


@pytest.mark.parametrize("lean", [False, True])
@pytest.mark.parametrize("pair,open_shell,iexch", CASES)
def test_one_and_two_shell_slots(pair, open_shell, iexch, lean):
    wl = molecule(pair, open_shell, iexch)
    assert wl.basis.M == 96
    options = dict(aaf=True)
    P = H.lib(H.os.path.join(H.ROOT, "lio_b200", "libg2g_b200.so"), True)
    P.set_lean(lean)
    try:
        E, K, Kb = H.run(P, wl, options=options, precision=1)
        _, F = P.solve_forces(2)
    finally:
        P.set_lean(False)
    E_ref, K_ref, Kb_ref, _ = H.restatement(wl, options=options)
    assert abs(E - E_ref) <= H.E_TOL
    assert np.max(np.abs(K - K_ref)) <= H.K_TOL
    if open_shell:
        assert np.max(np.abs(Kb - Kb_ref)) <= H.K_TOL
    _, F_ref, _ = H.restatement(wl, options=options, forces=True)
    assert np.max(np.abs(F - F_ref)) <= F_TOL
    print(pair, open_shell, E - E_ref, np.max(np.abs(K - K_ref)), np.max(np.abs(F - F_ref)), np.max(np.abs(K_ref)))
