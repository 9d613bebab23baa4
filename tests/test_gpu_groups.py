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
