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


def _context(n):
    from megadock_b200 import FFTProcess
    ng, gw = n // 2, 1.2
    length = np.float32(gw) * np.float32(ng)
    gc = (float(length) * (-0.5 + (0.5 + np.arange(ng)) / ng)).astype(np.float32)
    fp = FFTProcess(0)
    fp.alloc_array(n, gw, gc)
    return fp, gc


@pytest.mark.parametrize("n", [48, 128, 162])
@pytest.mark.parametrize("na,scale", [(20000, 1.0), (32768, 1.0), (32768, 4.0)])
def test_dense_planes_bit_exact(built, gpu, n, na, scale):
    """Planes with more charges than the shared list: a ball of atoms that fills
    the grid, and one four times as wide, whose charges are clamped to the
    outer planes and cells."""
    from megadock_b200 import rotation_matrix
    from oracle import oracle as O
    rng = np.random.default_rng(na + n)
    v = rng.normal(size=(na, 3))
    xyz = (v / np.linalg.norm(v, axis=1)[:, None] * rng.uniform(0, 1, (na, 1)) ** (1 / 3) * (0.6 * n / 2 * scale))
    xyz = xyz.astype(np.float32)
    _, rad, q = _ligand(na, False, n)
    fp, gc = _context(n)
    fp.ligand_data_transfer_gpu(xyz, rad, q)
    m = rotation_matrix(np.asarray((0.3, 1.1, 4.0), np.float32))
    dr, di = fp.ligand_voxels(m)
    gr, gi = O.ligand_grids(O.rotate(xyz, m), rad, q, n // 2, 1.2, gc, 1.0)
    assert np.array_equal(dr, gr) and np.array_equal(di, gi)


def test_dense_planes_take_time_by_the_atom(built, gpu):
    """The voxelizer stage of 32,768 atoms in a ball of 70 A at N = 128 (a grid of
    77 A) takes 3.5 times as long as that of 8,192 (12 when each cell walked all
    of its plane's charges)."""
    import torch

    from megadock_b200 import rotation_matrix
    ms = {}
    for na in (8192, 32768):
        rng = np.random.default_rng(7)
        v = rng.normal(size=(na, 3))
        xyz = v / np.linalg.norm(v, axis=1)[:, None] * rng.uniform(0, 1, (na, 1)) ** (1 / 3) * 70
        _, rad, q = _ligand(na, False, 1)
        fp, _ = _context(128)
        zero = np.zeros((64,) * 3, np.float32)
        fp.receptor_fft(zero, zero)
        fp.ligand_data_transfer_gpu(xyz.astype(np.float32), rad, q)
        d_rot = torch.from_numpy(rotation_matrix(np.zeros(3, np.float32)).reshape(-1)).cuda()
        d_out = torch.zeros(5, dtype=torch.int32, device="cuda")
        ms[na] = min(float(fp.dock_profile(d_rot.data_ptr(), 0, 1, 1, d_out.data_ptr())[0][0]) for _ in range(10))
    print(f"voxelizer stage: {ms}")
    assert ms[32768] < 6 * ms[8192], ms
