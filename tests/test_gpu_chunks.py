"""Kohn-Sham contraction split over a group's points (tensor-core form): chunks
of one 128-point tile, uneven chunks of one large group (also above 128
functions: two row tiles, and few rows: several K steps per copy), one and two
spins, with and without the blocked basis, against the C restatement at the
parity tolerances."""
import numpy as np
import pytest

from lio_b200 import workloads as W

from . import helpers as H

pytestmark = pytest.mark.gpu

CASES = [
    # (atoms, seed, open shell, little_cube_size, sphere_radius)
    (3, 301, False, 8.0, 0.6),    # fewer tiles than SMs: chunks of one tile
    (5, 302, True, 4.0, 0.0),     # many groups of one partial tile, 8 to 40 functions
    (16, 303, False, 40.0, 0.0),  # one group: every function, thousands of points
    (24, 304, True, 40.0, 0.3),   # the same above 128 functions, and small spheres
]


@pytest.mark.parametrize("lean", [False, True])
@pytest.mark.parametrize("atoms,seed,open_shell,lcs,sr", CASES)
def test_chunked_kohn_sham(atoms, seed, open_shell, lcs, sr, lean):
    wl = W.small_workload(atoms, seed, 9, open_shell, n_rad=20)
    options = dict(lcs=lcs, sr=sr)
    P = H.lib(H.os.path.join(H.ROOT, "lio_b200", "libg2g_b200.so"), True)
    P.set_lean(lean)
    try:
        E, K, Kb = H.run(P, wl, options=options, precision=1)
    finally:
        P.set_lean(False)
    E_ref, K_ref, Kb_ref, _ = H.restatement(wl, options=options)
    assert abs(E - E_ref) <= H.E_TOL
    assert np.max(np.abs(K - K_ref)) <= H.K_TOL
    if open_shell:
        assert np.max(np.abs(Kb - Kb_ref)) <= H.K_TOL
