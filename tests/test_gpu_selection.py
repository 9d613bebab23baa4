"""The inverse plane kernels and their top-t selection at the sizes where a
plan changes form (one CTA per plane, clusters of 2, 4 and 8, the warp-owned
form at 128) and at the list lengths where the selection does (the loose bound
up to 3 poses, the merged bound above, passes of 32)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-4, 1e-3   # FP32 transforms against FP64, as in test_gpu_parity.py


def _context(pairs, *extra):
    from megadock_b200 import FFTProcess, Job
    rp, lp = pairs["small"]
    job = Job(["-R", rp, "-L", lp, "-r", "360", *extra])
    fp = FFTProcess(0)
    fp.alloc_array(job.nf1, job.grid_width, job.grid_coord())
    xyz, rad, q = job.ligand_atoms()
    fp.ligand_data_transfer_gpu(xyz, rad, q, job.lig_core)
    return job, fp


@pytest.mark.parametrize("n", [48, 66, 96, 128, 150, 192, 242, 256, 330])
@pytest.mark.parametrize("t", [3, 4, 33])
def test_lists_are_prefixes_of_the_longest(built, gpu, pairs, n, t):
    """The t best poses of a rotation are the first t of its 70 best (three
    passes of the plane kernel), whichever bound and pass count found them,
    and one pose per rotation is the first of them."""
    from megadock_b200 import rotation_matrices
    gw = max(1.2, 1.2 * 96 / n)
    job, fp = _context(pairs, "-F", str(n), "-v", f"{gw:.3f}")
    rr, ri = job.receptor_grids()
    fp.receptor_fft(rr, ri)
    mats = rotation_matrices(job.rotation_angles()[:6])
    full = fp.cuda_fft(mats, t=70).copy().reshape(6, 70)
    assert np.array_equal(fp.cuda_fft(mats, t=t).reshape(6, t), full[:, :t])
    one = fp.cuda_fft(mats, t=1)
    up = full[:, 0]["score"] > 0
    assert np.array_equal(one[up], full[up, 0])
    s = full["score"]
    assert (s[:, 1:] <= s[:, :-1]).all()
    cells = (full["i"].astype(np.int64) * n + full["j"]) * n + full["k"]
    assert all(len(set(c)) == 70 for c in cells)


@pytest.mark.parametrize("n", [48, 128, 192, 256, 330])
@pytest.mark.parametrize("t", [1, 2, 5, 40])
def test_equal_scores_go_to_the_lowest_cells(built, gpu, pairs, n, t):
    """A receptor of zeros scores 0 everywhere: more equal keys than the
    shared list holds, and the answer is the first t cells in order."""
    from megadock_b200 import rotation_matrices
    job, fp = _context(pairs, "-F", str(n), "-v", f"{max(1.2, 1.2 * 96 / n):.3f}")
    zero = np.zeros((n // 2,) * 3, np.float32)
    fp.receptor_fft(zero, zero)
    got = fp.cuda_fft(rotation_matrices(job.rotation_angles()[:3]), t=t).reshape(3, t)
    assert (got["score"] == 0).all()
    cells = (got["i"].astype(np.int64) * n + got["j"]) * n + got["k"]
    assert (cells == np.arange(t)).all()


@pytest.mark.parametrize("n", [100, 144, 180, 252])
def test_long_lists_match_fp64(built, gpu, pairs, n):
    """Twelve poses per rotation against the FP64 oracle at one size of each
    cluster width (1, 1, 2, 8)."""
    from megadock_b200 import rotation_matrices
    from oracle import oracle as O
    job, fp = _context(pairs, "-F", str(n))
    rr, ri = job.receptor_grids()
    fp.receptor_fft(rr, ri)
    rhat = O.receptor_spectrum(rr, ri, n, "fp64")
    xyz, rad, q = job.ligand_atoms()
    mats = rotation_matrices(job.rotation_angles()[[0, 200]])
    got = fp.cuda_fft(mats, t=12).reshape(2, 12)
    for m, g in zip(mats, got):
        gr, gi = O.ligand_grids(O.rotate(xyz, m), rad, q, job.ng1, job.grid_width, job.grid_coord(), job.lig_core)
        raw = O.raw_scores(rhat, gr, gi, "fp64")
        want, _ = O.score_sort(raw.astype(np.float32), 12)
        assert np.all(np.abs(g["score"] - want) <= RTOL * np.abs(want) + ATOL)
        at = raw[g["i"], g["j"], g["k"]] / float(n) ** 3
        assert np.all(np.abs(g["score"] - at) <= RTOL * np.abs(at) + ATOL)


@pytest.mark.parametrize("n", [126, 162, 220, 252])
@pytest.mark.parametrize("t", [31, 150])
def test_merged_lists_match_fp64(built, gpu, pairs, n, t):
    """Lists longer than a pass, merged over 126 to 2,016 of them a rotation
    (fewer than, and several for each of, the merge's 256 threads)."""
    from megadock_b200 import rotation_matrices
    from oracle import oracle as O
    job, fp = _context(pairs, "-F", str(n))
    rr, ri = job.receptor_grids()
    fp.receptor_fft(rr, ri)
    xyz, rad, q = job.ligand_atoms()
    m = rotation_matrices(job.rotation_angles()[[123]])
    got = fp.cuda_fft(m, t=t)
    gr, gi = O.ligand_grids(O.rotate(xyz, m[0]), rad, q, job.ng1, job.grid_width, job.grid_coord(), job.lig_core)
    raw = O.raw_scores(O.receptor_spectrum(rr, ri, n, "fp64"), gr, gi, "fp64")
    want = np.sort(raw.reshape(-1))[::-1][:t] / float(n) ** 3
    assert np.all(np.abs(got["score"] - want) <= RTOL * np.abs(want) + ATOL)
    at = raw[got["i"], got["j"], got["k"]] / float(n) ** 3
    assert np.all(np.abs(got["score"] - at) <= RTOL * np.abs(at) + ATOL)
    assert len(set(zip(got["i"], got["j"], got["k"]))) == t


def test_merge_time_does_not_follow_the_lists(built, gpu, pairs):
    """A hundred poses of one rotation from 880 lists (N = 220, four CTAs per
    plane) merge in about the time of 160 lists (N = 160): a round compares the
    lists' heads.  Scanning every candidate in every round took 4 times as long."""
    import torch

    from megadock_b200 import rotation_matrices
    ms = {}
    for n in (160, 220):
        job, fp = _context(pairs, "-F", str(n))
        fp.receptor_fft(*job.receptor_grids())
        d_rot = torch.from_numpy(np.ascontiguousarray(rotation_matrices(job.rotation_angles()[:1]))).cuda()
        d_out = torch.zeros(100 * 5, dtype=torch.int32, device="cuda")
        ms[n] = min(float(fp.dock_profile(d_rot.data_ptr(), 0, 1, 100, d_out.data_ptr())[0][4]) for _ in range(8))
    print(f"merge of 100 poses: {ms}")
    assert ms[220] < 2 * ms[160], ms


def test_overflowing_lists_are_bounded_again(built, gpu, pairs):
    """N = 96, where 32 poses let more cells through the first bound than the
    shared list holds: the stage takes 1.8 times as long as for 3 poses (3.1
    when every cell was then found by a round of its own)."""
    import torch

    from megadock_b200 import rotation_matrices
    job, fp = _context(pairs, "-F", "96")
    fp.receptor_fft(*job.receptor_grids())
    fp.set_batch(32)
    d_rot = torch.from_numpy(np.ascontiguousarray(rotation_matrices(job.rotation_angles()[:32]))).cuda()
    d_out = torch.zeros(32 * 32 * 5, dtype=torch.int32, device="cuda")
    ms = {t: min(float(fp.dock_profile(d_rot.data_ptr(), 0, 32, t, d_out.data_ptr())[0][3]) for _ in range(10))
          for t in (3, 32)}
    print(f"inverse planes of 32 rotations: {ms}")
    assert ms[32] < 2.4 * ms[3], ms
