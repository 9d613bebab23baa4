"""A context that was never given rotations per launch groups them itself: the
records are the plain form's, bit for bit, at one rotation, below, at and above
one group, and for the other entry points that launch in groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,counts", [(48, (1, 2, 64, 65, 200)), (128, (1, 51, 120)), (256, (1, 9))])
@pytest.mark.parametrize("t", [1, 3])
def test_automatic_groups_equal_plain(built, gpu, pairs, n, counts, t):
    from megadock_b200 import FFTProcess, Job, rotation_matrices
    rp, lp = pairs["small"]
    job = Job(["-R", rp, "-L", lp, "-r", "360", "-F", str(n), "-v", f"{max(1.2, 1.2 * 96 / n):.3f}"])

    def context():
        fp = FFTProcess(0)
        fp.alloc_array(job.nf1, job.grid_width, job.grid_coord())
        fp.receptor_fft(*job.receptor_grids())
        xyz, rad, q = job.ligand_atoms()
        fp.ligand_data_transfer_gpu(xyz, rad, q, job.lig_core)
        return fp

    auto, plain = context(), context()
    plain.set_batch(1)
    mats = rotation_matrices(job.rotation_angles())
    for c in counts:
        a = auto.cuda_fft(mats[:c], t=t, first_rot=7).copy()
        assert np.array_equal(a, plain.cuda_fft(mats[:c], t=t, first_rot=7)), c
    k = counts[-1]
    poses = auto.cuda_fft(mats[:k], t=1).copy()
    assert np.array_equal(auto.pose_scores(mats[:k], poses), plain.pose_scores(mats[:k], poses))
    w = np.linspace(-1, 1, k).astype(np.float32)
    ga, gp = auto.adjoint_poses(mats[:k], poses, w), plain.adjoint_poses(mats[:k], poses, w)
    assert all(np.array_equal(ga[key], gp[key]) for key in ("d_rec_r", "d_rec_i", "d_charge"))


@pytest.mark.parametrize("n", [48, 128, 256])
def test_callers_graph_outlives_larger_calls(built, gpu, pairs, n):
    """A caller captures md_dock_device on its own stream; after calls that need
    larger work buffers the graph still replays to the same records."""
    import torch

    from megadock_b200 import POSE_DTYPE, FFTProcess, Job, rotation_matrices
    rp, lp = pairs["small"]
    job = Job(["-R", rp, "-L", lp, "-r", "360", "-F", str(n), "-v", f"{max(1.2, 1.2 * 96 / n):.3f}"])
    s = torch.cuda.Stream()
    fp = FFTProcess(0, stream=s.cuda_stream)
    fp.alloc_array(job.nf1, job.grid_width, job.grid_coord())
    fp.receptor_fft(*job.receptor_grids())
    xyz, rad, q = job.ligand_atoms()
    fp.ligand_data_transfer_gpu(xyz, rad, q, job.lig_core)
    mats = rotation_matrices(job.rotation_angles())
    want = fp.cuda_fft(mats[:5], t=2).copy()
    d_rot = torch.from_numpy(np.ascontiguousarray(mats[:5], np.float32)).cuda()
    d_out = torch.zeros(5 * 2 * 5, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        fp.dock_device(d_rot.data_ptr(), 0, 5, 2, d_out.data_ptr())

    def replayed():
        with torch.cuda.stream(s):
            d_out.zero_()
            graph.replay()
        torch.cuda.synchronize()
        return d_out.cpu().numpy().view(POSE_DTYPE)

    assert np.array_equal(replayed(), want)
    many = fp.cuda_fft(mats[:120], t=2).copy()
    assert np.array_equal(replayed(), want)
    fp.pose_scores(mats[:120], fp.cuda_fft(mats[:120], t=1))
    fp.cuda_fft(mats[:2], t=40)
    assert np.array_equal(replayed(), want)
    assert np.array_equal(fp.cuda_fft(mats[:120], t=2), many)


def test_pairs_of_default_contexts(built, gpu, tmp_path):
    """Pair contexts without a launch size group their rotations too."""
    import ctypes as C

    import torch

    from megadock_b200 import POSE_DTYPE, FFTProcess, Job, lib, rotation_matrices, synth
    t, k = 2, 70
    ctxs, plain = [], []
    for nr, nl, seed, n in [(30, 16, 8, 64), (60, 40, 32, 84), (30, 16, 9, 180)]:
        rp, lp = synth.write_pair(str(tmp_path), nr, nl, seed, stem=f"d{seed}")
        job = Job(["-R", rp, "-L", lp, "-r", "360", "-F", str(n)])
        mats = rotation_matrices(job.rotation_angles())[:k]
        for out in (ctxs, plain):
            fp = FFTProcess(0)
            fp.alloc_array(job.nf1, job.grid_width, job.grid_coord())
            job.receptor_to(fp)
            xyz, rad, q = job.ligand_atoms()
            fp.ligand_data_transfer_gpu(xyz, rad, q, job.lig_core)
            out.append(fp)
    d_rot = torch.from_numpy(np.ascontiguousarray(mats)).cuda()
    d_out = [torch.zeros(k * t * 5, dtype=torch.int32, device="cuda") for _ in ctxs]
    torch.cuda.synchronize()
    runner, m = FFTProcess(0), len(ctxs)
    rc = lib().md_dock_pairs(runner._h, (C.c_void_p * m)(*[fp._h.value for fp in ctxs]), m,
                             (C.c_void_p * m)(*[d_rot.data_ptr()] * m), (C.c_int * m)(*[k] * m), t,
                             (C.c_void_p * m)(*[o.data_ptr() for o in d_out]))
    assert rc == 0
    torch.cuda.synchronize()
    for fp, o in zip(plain, d_out):
        fp.set_batch(1)
        assert np.array_equal(o.cpu().numpy().view(POSE_DTYPE), fp.cuda_fft(mats, t=t))
