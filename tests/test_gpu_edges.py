"""Both forms at the edges of the contractions' tiles: groups from one shell to all
functions of a molecule (8-, 16-, 32- and 64-function edges, shells that straddle
an epilogue window), partial 64- and 128-point tiles, one to many chunks of a
group's points; energy, Kohn-Sham matrices and forces against the C restatement at
the parity tolerances."""
import numpy as np
import pytest

from lio_b200 import workloads as W

from . import helpers as H

pytestmark = pytest.mark.gpu

F_TOL = 1e-7  # Hartree / bohr, as the parity tests of the forces

CASES = [
    # (atoms, seed, iexch, open shell, little_cube_size, sphere_radius)
    (3, 401, 3, False, 4.0, 0.6),
    (7, 402, 9, True, 5.0, 0.3),
    (13, 403, 3, False, 40.0, 0.0),
    (18, 404, 9, False, 40.0, 0.0),
    (21, 405, 9, True, 6.0, 0.6),
]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("atoms,seed,iexch,open_shell,lcs,sr", CASES)
def test_tile_edges(atoms, seed, iexch, open_shell, lcs, sr, precision):
    wl = W.small_workload(atoms, seed, iexch, open_shell, n_rad=20)
    options = dict(lcs=lcs, sr=sr)
    P = H.lib(H.os.path.join(H.ROOT, "lio_b200", "libg2g_b200.so"), True)
    E, K, Kb = H.run(P, wl, options=options, precision=precision)
    _, F = P.solve_forces(2)
    E_ref, K_ref, Kb_ref, _ = H.restatement(wl, options=options)
    assert abs(E - E_ref) <= H.E_TOL
    assert np.max(np.abs(K - K_ref)) <= H.K_TOL
    if open_shell:
        assert np.max(np.abs(Kb - Kb_ref)) <= H.K_TOL
    _, F_ref, _ = H.restatement(wl, options=options, forces=True)
    assert np.max(np.abs(F - F_ref)) <= F_TOL
