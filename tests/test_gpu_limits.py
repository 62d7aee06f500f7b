"""Limits of the tensor-core form that the engine enforces on the host.

A grid whose cubes are large enough to hold a group of more than 87,296 padded
points (here one cube for the whole molecule, through little_cube_size), or a
group of more functions than the form's limit (2,912 at closed-shell GGA), must
be refused with a clear error, before any kernel runs, while the FP64 form still
builds it. The messages give the limit and no reason that the kernels no longer
have: their accumulators and shared memory hold more than either limit."""
import numpy as np
import pytest

from lio_b200 import workloads as W

from . import helpers as H


@pytest.mark.gpu
def test_tensor_core_refuses_a_group_above_its_accumulator_limit():
    wl = W.small_workload(24, 5, 9, False)
    L = H.lib(H.os.path.join(H.ROOT, "lio_b200", "libg2g_b200.so"), True)
    gt = H.bind(L, wl, options=dict(lcs=1000.0, sr=0.0))  # every point in one cube
    L.set_precision(1)
    msg = L.reload_atom_positions(gt)
    assert not msg, msg
    st = L.partition_stats()
    big = max(L.partition_group(g)["meta"][0] for g in range(st["groups"]))
    assert big > 87296, big
    with pytest.raises(RuntimeError, match="exceeds its limit"):
        L.solve_groups(0)
    L.set_precision(0)
    E = L.solve_groups(0)
    assert np.isfinite(E)
    L.deinit()


def many_functions(m):
    """One hydrogen with m s functions on a small grid: one group of m functions."""
    mol = W.Molecule(["H"], np.array([1]), np.zeros((1, 3)))
    shells = [(0, 1, 0.1 * 1.003 ** k) for k in range(m)]
    q = W.random_orbitals(m, 2, np.random.default_rng(4))
    return H.shells_workload(mol, shells, W.pack_lower(2.0 * q @ q.T, True), 9, False, n_rad=1)


@pytest.mark.gpu
def test_tensor_core_refuses_a_group_above_its_function_limit():
    L = H.lib(H.os.path.join(H.ROOT, "lio_b200", "libg2g_b200.so"), True)
    options = dict(lcs=1000.0, sr=0.0)
    # the largest accepted
    wl = many_functions(2912)
    E, K, _ = H.run(L, wl, options=options, precision=1)
    assert L.partition_group(0)["meta"][5] == 2912
    E_ref, K_ref, _, _ = H.restatement(wl, options=options)
    assert abs(E - E_ref) <= H.E_TOL
    assert np.max(np.abs(K - K_ref)) <= H.K_TOL
    # one more
    gt = H.bind(L, many_functions(2913), options=options)
    L.set_precision(1)
    assert not L.reload_atom_positions(gt)
    with pytest.raises(RuntimeError, match="2913 functions exceeds its limit of 2912") as e:
        L.solve_groups(0)
    assert "shared memory" not in str(e.value)
    L.set_precision(0)
    assert np.isfinite(L.solve_groups(0))
    L.deinit()
