"""Receptor grids where the bit-mask form can go wrong: one to four mask words
and the edges between them, core values that collide with the markers' meaning
(0 makes every cell core), no electrostatics, a single atom, atoms off the
grid, more atoms near a row than the shared list holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(pairs, *extra):
    from megadock_b200 import FFTProcess, Job
    rp, lp = pairs["c0"]
    job = Job(["-R", rp, "-L", lp, *extra])
    fp = FFTProcess(0)
    fp.alloc_array(job.nf1, job.grid_width, job.grid_coord())
    xyz, rad, q, ace = job.receptor_atoms()
    rc, _ = job.centers()
    return job, fp, (xyz.reshape(-1, 3) - np.asarray(rc, np.float32)).astype(np.float32), rad, q, ace


@pytest.mark.parametrize("extra,core,acer,elec", [
    (("-F", "126"), -45.0, 1.0, 1.0),                                    # ng1 = 63, 64, 65: the first word's edge
    (("-F", "128"), -45.0, 1.0, 1.0),
    (("-F", "132", "-a", "3"), 3.0, 1.0, 1.0),                           # a positive core value
    (("-F", "252", "-v", "0.7"), -45.0, 1.0, 1.0),                       # 126, 128, 130
    (("-F", "256", "-v", "0.55", "-e", "0"), -45.0, 1.0, 0.0),
    (("-F", "384", "-v", "0.5"), -45.0, 1.0, 1.0),                       # 192 and 196: three words, four
    (("-F", "392", "-v", "0.5"), -45.0, 1.0, 1.0),
    (("-F", "64", "-v", "1.9", "-a", "0"), 0.0, 1.0, 1.0),               # every cell compares equal to the core
])
def test_grids_bit_exact(built, gpu, pairs, extra, core, acer, elec):
    job, fp, xyz, rad, q, ace = _case(pairs, *extra)
    hr, hi = job.receptor_grids()
    dr, di = fp.receptor_build(xyz, rad, q, ace, core, acer, elec, make_receptor=False, return_grids=True)
    assert np.array_equal(dr, hr), f"{(dr != hr).sum()} real cells differ"
    assert np.array_equal(di, hi), f"{(di != hi).sum()} field cells differ"


def test_repeated_builds_share_scratch(built, gpu, pairs):
    """A larger build, a smaller one and the larger again in one context give
    what fresh contexts give (the masks and atom records are cleared or
    rewritten by every call), and one atom or atoms off the grid are taken."""
    _, fp, xyz, rad, q, ace = _case(pairs, "-F", "128")
    cases = [(xyz, rad, q, ace), (xyz[:1], rad[:1], q[:1], ace[:1]), (xyz * 2 + 9, rad, q, ace), (xyz, rad, q, ace)]
    got = [fp.receptor_build(*c, make_receptor=False, return_grids=True) for c in cases]
    for c, g in zip(cases, got):
        _, one, *_ = _case(pairs, "-F", "128")
        want = one.receptor_build(*c, make_receptor=True, return_grids=True)
        assert np.array_equal(g[0], want[0]) and np.array_equal(g[1], want[1])
    assert np.array_equal(got[0][0], got[3][0])
