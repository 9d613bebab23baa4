"""Work buffers of a context on the CPU: the library's host side linked against
a CUDA runtime without a device (tests/fake_runtime), whose device memory is a
ledger under a budget.  Covers what no run on a GPU shows without a fault or an
exhausted device: which buffers a captured launch keeps using, what a context
does where its automatic launch groups have no room."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "megadock_b200" / "csrc"
FAKE = ROOT / "tests" / "fake_runtime"
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
MIB = 1 << 20


@pytest.fixture(scope="module")
def rt(tmp_path_factory):
    """md_b200.cu and the fake runtime as one library (device code as PTX only)."""
    if not Path(NVCC).exists():
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("fake")
    flags = [NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=compute_100a",
             "-Xcompiler", "-fPIC,-fno-gnu-unique", "-c"]   # nothing shared with the real library
    jobs = [subprocess.Popen(flags + ["-o", str(d / f"{src.stem}.o"), str(src)], stderr=subprocess.PIPE, text=True)
            for src in (CSRC / "md_b200.cu", FAKE / "fake_sizes.cu", FAKE / "fake_runtime.cpp")]
    for j in jobs:
        _, err = j.communicate()
        assert j.returncode == 0, err
    so = d / "libfake.so"
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", str(so), *map(str, d.glob("*.o"))], check=True)
    lib = C.CDLL(str(so))
    from megadock_b200._native import _PROTOS
    for name, (res, args) in _PROTOS.items():
        if hasattr(lib, name):
            getattr(lib, name).restype, getattr(lib, name).argtypes = res, args
    lib.fake_used.restype = C.c_size_t
    lib.fake_budget.argtypes = [C.c_size_t]
    return lib


class Context:
    """A context with a grid, a receptor and a ligand of 20 atoms."""

    def __init__(self, rt, n, batch=0, device=0):
        self.rt, self.n = rt, n
        self.h = C.c_void_p()
        assert rt.md_ctx_create(device, C.byref(self.h)) == 0
        ng = n // 2
        z = np.zeros(ng ** 3)
        self.ok(rt.md_set_grid(self.h, n, 1.2, _f(np.arange(ng))))
        if batch:
            self.ok(rt.md_set_batch(self.h, batch))
        self.ok(rt.md_receptor_fft(self.h, _f(z), _f(z)))
        a = np.ones(60)
        self.ok(rt.md_ligand_data(self.h, 20, _f(a), _f(a), _f(a), 1.0))

    def ok(self, rc):
        assert rc == 0, self.rt.md_last_error(self.h).decode()

    def dock(self, n, t=1):
        out = np.zeros(5 * n * t, np.int32)
        self.ok(self.rt.md_dock(self.h, _f(np.zeros(9 * n)), 0, n, t, out.ctypes.data))

    def dock_device(self, n, t=1):
        self.ok(self.rt.md_dock_device(self.h, C.c_void_p(1 << 20), 0, n, t, C.c_void_p(1 << 21)))

    def pose_scores(self, n):
        poses = np.zeros(5 * n, np.int32)
        self.ok(self.rt.md_pose_scores(self.h, _f(np.zeros(9 * n)), n, poses.ctypes.data, _f(np.zeros(n))))

    def profile(self, n, t=1):
        self.ok(self.rt.md_dock_profile(self.h, C.c_void_p(1 << 20), 0, n, t, C.c_void_p(1 << 21), _f(np.zeros(5)),
                                        None))

    def pose_terms(self, n):
        tem = np.zeros(3 * n, np.int32)
        self.ok(self.rt.md_pose_terms(self.h, _f(np.zeros((self.n // 2) ** 3)), _f(np.zeros(9 * n)), n,
                                      tem.ctypes.data_as(C.POINTER(C.c_int)), _f(np.zeros(9 * n))))

    def adjoint(self, n):
        poses = np.zeros(5 * n, np.int32)
        ng3 = (self.n // 2) ** 3
        self.ok(self.rt.md_adjoint_poses(self.h, _f(np.zeros(9 * n)), n, poses.ctypes.data, _f(np.ones(n)),
                                         _f(np.zeros(ng3)), _f(np.zeros(ng3)), _f(np.zeros(20)), None, 0, None, None))

    def pairs(self, others, n, t=1):
        k = len(others)
        rots, outs = (C.c_void_p * k)(*[1 << 20] * k), (C.c_void_p * k)(*[1 << 21] * k)
        self.ok(self.rt.md_dock_pairs(self.h, (C.c_void_p * k)(*[o.h.value for o in others]), k, rots,
                                      (C.c_int * k)(*[n] * k), t, outs))

    def capture(self, n, t=1):
        """The launches of md_dock_device on a stream the caller is capturing."""
        first = self.rt.fake_launches()
        self.rt.fake_capture(1)
        self.dock_device(n, t)
        self.rt.fake_capture(0)
        return range(first, self.rt.fake_launches())

    def close(self):
        self.rt.md_ctx_destroy(self.h)


def _f(a):
    return np.ascontiguousarray(a, np.float32).ctypes.data_as(C.POINTER(C.c_float))


@pytest.fixture
def context(rt):
    made = []

    def make(*a, **k):
        made.append(Context(rt, *a, **k))
        return made[-1]

    rt.fake_budget(1 << 62)
    yield make
    rt.fake_capture(0)
    for c in made:
        c.close()
    rt.fake_forget()
    assert rt.fake_used() == 0
    assert rt.fake_short() == 0   # no launch got freed or too small buffers


@pytest.mark.parametrize("batch", [0, 1])
@pytest.mark.parametrize("n", [48, 128, 256])
def test_captured_launches_keep_their_buffers(rt, context, n, batch):
    """What a caller captured stays valid through later calls that need larger
    buffers (more rotations, poses per rotation, rotations per launch), and
    until the caller gives the work buffers back."""
    c = context(n, batch)
    c.dock(2)
    held = list(c.capture(5))
    larger = [lambda: c.dock(200), lambda: c.dock(3, t=40), lambda: c.pose_scores(64)]
    for call in larger:
        call()
        held += c.capture(4)
    c.ok(rt.md_set_batch(c.h, 300))
    c.dock(300)
    assert len(held) > 4 and all(rt.fake_live(k) for k in held)
    c.ok(rt.md_release_work(c.h))
    assert not any(rt.fake_live(k) for k in held)
    c.dock(2)


def test_captured_launches_survive_a_failed_growth(rt, context):
    c = context(48)
    c.dock(2)
    held = c.capture(2)
    rt.fake_budget(rt.fake_used() + 1 * MIB)
    c.dock(100)
    c.pose_scores(20)
    assert all(rt.fake_live(k) for k in held)


def test_uncaptured_work_buffers_do_not_add_up(rt, context):
    """Without a capture a growing call replaces the buffers."""
    a, b = context(48), context(48)
    before = rt.fake_used()
    for n in (1, 2, 7, 40, 64):
        a.dock(n)
    grown = rt.fake_used() - before
    before = rt.fake_used()
    b.dock(64)
    assert grown == rt.fake_used() - before


# one rotation of the work set at N = 128: 2 x 8 ng N^2 bytes and the charge lists
ONE_128 = 2 * 8 * 64 * 128 * 128 + 8 * 64 ** 3


@pytest.mark.parametrize("call,sets,extra", [
    (lambda c: c.dock(200), 1, 0),
    (lambda c: c.dock_device(200), 1, 0),
    (lambda c: c.profile(200), 1, 0),
    (lambda c: c.pose_scores(200), 1, 8 * 64 ** 3),
    (lambda c: c.adjoint(200), 1, 2 * 8 * 64 ** 3),
    (lambda c: c.pose_terms(200), 1, 201 * 8 * 64 ** 3),   # its own voxel grids: 200 poses
    (lambda c: c.pairs([c, c], 200), 2, 0),
])
def test_automatic_groups_fall_back_to_one_rotation(rt, context, call, sets, extra):
    """Every call that groups rotations by itself still runs where there is room
    for one rotation only, does not ask for the large buffers again in later
    calls, and groups again after md_release_work."""
    c = context(128)
    c.ok(rt.md_release_work(c.h))
    free = rt.fake_used()
    rt.fake_budget(free + sets * ONE_128 + extra + 4 * MIB)
    rt.fake_forget()
    call(c)
    assert {rt.fake_rotations(k) for k in range(rt.fake_launches())} == {1}
    refused = rt.fake_refused()
    call(c)
    assert rt.fake_refused() == refused
    rt.fake_budget(1 << 62)
    c.ok(rt.md_release_work(c.h))
    rt.fake_forget()
    call(c)
    assert max(rt.fake_rotations(k) for k in range(rt.fake_launches())) > 1


def test_no_room_for_one_rotation_is_an_error(rt, context):
    """... after which the same call runs once there is room."""
    c = context(128)
    c.ok(rt.md_release_work(c.h))
    rt.fake_budget(rt.fake_used() + ONE_128 // 2)
    for call in (c.dock, c.dock_device, c.profile, c.pose_scores, c.pose_terms, lambda n: c.pairs([c], n)):
        with pytest.raises(AssertionError, match="out of memory"):
            call(100)
    rt.fake_budget(1 << 62)
    for call in (c.dock, c.dock_device, c.profile, c.pose_scores, c.pose_terms, lambda n: c.pairs([c], n)):
        rt.fake_forget()
        call(100)
        assert rt.fake_rotations(0) > 1


@pytest.mark.parametrize("n", [48, 128, 256])
def test_kernel_attributes_are_set_on_every_device(rt, context, n):
    """The shared-memory opt-in of a size's kernels belongs to one device: a
    second device's context of that size sets it too, once."""
    context(n, device=0)
    before = rt.fake_attrs(1)
    context(n, device=1)
    own = rt.fake_attrs(1) - before
    assert own > 0
    rt.fake_attr_calls(1)
    context(n, device=1)
    assert rt.fake_attr_calls(0) == 0


@pytest.mark.parametrize("n,per_plane", [(48, 1), (128, 1), (256, 8)])
def test_candidate_lists_hold_one_per_cta(rt, context, n, per_plane):
    """Candidate lists of a launch group: 8 bytes a pose for each CTA that
    selects (one per x plane up to N = 160, a cluster's CTAs above)."""
    a, b = context(n, batch=8), context(n, batch=8)
    for c in (a, b):
        c.ok(rt.md_set_lanes(c.h, 1))   # one work set
    before = rt.fake_used()
    a.dock(8, t=1)
    one = rt.fake_used() - before
    before = rt.fake_used()
    b.dock(8, t=501)
    poses = 500 * 8 * 20   # the host call's pose records
    assert rt.fake_used() - before - one == 500 * 8 * 8 * n * per_plane + poses


@pytest.mark.parametrize("n,own", [(48, ()), (128, (1,)), (256, ())])
def test_settings_that_select_no_other_kernel_keep_graphs(rt, context, n, own):
    """Only a plan with a kernel of its own drops the captured graphs."""
    c = context(n, batch=4)
    c.dock(8)
    graphs = rt.fake_graphs()
    for tile in (8, 16, 32):
        c.ok(rt.md_set_tile(c.h, tile))
    for plan in (2, 1, 2, 0):
        c.ok(rt.md_set_plan(c.h, plan))
        if plan not in own:
            c.dock(8)
    c.dock(8)
    assert rt.fake_graphs() == graphs + 1 if own else rt.fake_graphs() == graphs
    assert rt.md_set_tile(c.h, 12) and rt.md_set_plan(c.h, 3) and rt.md_set_plan(c.h, -1)   # still refused


@pytest.mark.parametrize("n", [48, 128])
def test_repeated_small_calls_allocate_nothing(rt, context, n):
    """The second of two equal calls finds its buffers in place; a call that
    needed hundreds of MB gives them back."""
    c = context(n)
    g = np.zeros((n // 2) ** 3, np.float32)
    for call in (lambda: c.ok(rt.md_ligand_voxels(c.h, _f(np.zeros(9)), _f(g), _f(g))), lambda: c.pose_terms(3),
                 lambda: c.pose_scores(3), lambda: c.adjoint(3), lambda: c.dock(3)):
        call()
        made = rt.fake_mallocs()
        call()
        assert rt.fake_mallocs() == made
    c.dock(6400)   # the work set at its largest group
    before = rt.fake_used()
    many = (200 << 20) // (8 * (n // 2) ** 3)
    c.pose_terms(many)
    assert rt.fake_used() <= before
