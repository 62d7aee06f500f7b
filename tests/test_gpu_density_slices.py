"""The gradient kinds' half of the density in the tensor-core form.

The density stage contracts dF/dx, dF/dy and dF/dz with the part of the density
D before the diagonal of each 32-function tile, the tile's own strict triangle
included, and half of the diagonal. The off-diagonal entries must keep every
digit that the full slices keep. Here they are one unit of the tile's last
digit: one function, too tight to reach any grid point, carries the density
2^40, which alone sets the tile's exponent; every other pair of functions has
the density 1 (the unit), the diagonal 2. With 2^39 in its place the same
entries are two units. Both products are exact integers, so the two builds may
differ by the order of the Kohn-Sham sums alone; entries cut on a grid one bit
coarser would round to 0 in the first and stay in the second."""
import numpy as np
import pytest

from lio_b200 import workloads as W

from . import helpers as H

pytestmark = pytest.mark.gpu


def one_tile_molecule(open_shell, big):
    """Five hydrogens with two s and one p shell each and one tight s: 26 functions, one tile."""
    mol = W.random_cluster({"H": 5}, 2.0, 11)
    # exp(-a r^2) is dropped where a r^2 > 70: beyond 3e-4 bohr, inside the innermost radial shell
    shells = [(0, 1, 1.0e9)]
    for atom in range(1, 6):
        shells += [(0, atom, 1.4), (0, atom, 0.35), (1, atom, 0.6)]
    D = np.ones((26, 26)) + np.eye(26)
    D[0, :] = D[:, 0] = 0.0  # function 0 is the tight one
    D[0, 0] = big
    return H.shells_workload(mol, shells, W.pack_lower(D, True), 9, open_shell, n_rad=30)


@pytest.mark.parametrize("open_shell", [False, True])
def test_off_diagonal_entries_of_the_diagonal_block_keep_their_last_digit(open_shell):
    P = H.lib(H.os.path.join(H.ROOT, "lio_b200", "libg2g_b200.so"), True)
    options = dict(aaf=True)  # every function in every group: one tile, one exponent
    K = {}
    for big in (2.0 ** 40, 2.0 ** 39):
        _, K[big], _ = H.run(P, one_tile_molecule(open_shell, big), options=options, precision=1)
    _, K_ref, _, _ = H.restatement(one_tile_molecule(open_shell, 1.0), options=options)
    scale = np.linalg.norm(K_ref)
    # the unit meets the basis values' leading digit alone, 2^-8 of the largest value; that is no more than a check
    # that the inputs mean what is said above
    assert np.linalg.norm(K[2.0 ** 39] - K_ref) <= 2.0 ** -5 * scale
    diff = np.linalg.norm(K[2.0 ** 40] - K[2.0 ** 39]) / scale
    print(open_shell, diff, np.linalg.norm(K[2.0 ** 39] - K_ref) / scale)
    # FP64 sums of some 10^4 points in another order
    assert diff <= 1e-12
