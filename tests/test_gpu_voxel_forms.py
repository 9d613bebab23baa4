"""The atom preparation and charge sums at the sizes where they change form:
ligands around the wide block's threshold, atom runs that do not fill a step,
planes that hold more charges than the shared list, cells with many charges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ligand(na, flat, seed):
    rng = np.random.default_rng(seed)
    xyz = rng.uniform(-1, 1, (na, 3)) * (1.0 if flat else 22.0)
    if flat:   # every charge in a few cells of two planes
        xyz[:, 0] = rng.choice([-0.3, 0.3], na)
    rad = rng.choice(np.array([1.48, 1.67, 2.02], np.float32), na)
    q = rng.choice(np.array([0.0, -0.57, 0.1, 0.25], np.float32), na)
    return xyz.astype(np.float32), rad.astype(np.float32), q.astype(np.float32)


@pytest.mark.parametrize("n", [64, 330, 420])
@pytest.mark.parametrize("na,flat", [(1, False), (33, False), (3072, False), (3073, False), (5000, False), (700, True),
                                     (4000, True)])
def test_voxels_bit_exact(built, gpu, n, na, flat):
    from megadock_b200 import FFTProcess, rotation_matrix
    from oracle import oracle as O
    ng, gw = n // 2, 1.2
    length = np.float32(gw) * np.float32(ng)
    gc = (float(length) * (-0.5 + (0.5 + np.arange(ng)) / ng)).astype(np.float32)
    xyz, rad, q = _ligand(na, flat, na + n)
    fp = FFTProcess(0)
    fp.alloc_array(n, gw, gc)
    fp.ligand_data_transfer_gpu(xyz, rad, q)
    for theta in ((0.0, 0.0, 0.0), (0.3, 1.1, 4.0)):
        m = rotation_matrix(np.asarray(theta, np.float32))
        dr, di = fp.ligand_voxels(m)
        gr, gi = O.ligand_grids(O.rotate(xyz, m), rad, q, ng, gw, gc, 1.0)
        assert np.array_equal(dr, gr) and np.array_equal(di, gi), theta
