"""Performance cases of the docking framework: what a user's program has it do.

Every case goes through the public Python interface (``FFTProcess`` and, for
the many-pairs form, the C ABI's ``md_dock_pairs``) with the buffers and
settings such a program keeps.  Molecules are random ellipsoids of atoms at
protein density whose long axis follows MEGADOCK's automatic grid sizing
(receptor extent + 16 A at 1.2 A per cell), so every grid is filled the way an
automatically sized job fills it.

``listed`` gives the fixed cases, ``draw`` more of the same ranges, ``exact``
the outputs in 64 bits from plain torch.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from megadock_b200 import FFTProcess
from megadock_b200._native import POSE_DTYPE, lib

GRID_WIDTH = 1.2                       # MEGADOCK's default -v
RADII = np.array([1.48, 1.38, 1.54, 1.67, 2.02, 1.63, 1.82, 1.99], np.float32)       # CHARMM table values
CHARGES = np.array([0.0, 0.0, 0.0, -0.57, 0.10, -0.25, -0.15, -0.55, 0.60, 0.25], np.float32)
ATOM_VOLUME = 18.0                     # A^3 per heavy atom of a protein
MAX_LIGAND_ATOMS = 12000


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: one orientation of a peptide scored on a small grid with a
        # fresh context's settings, where launches and copies are everything
        dict(name="single-48", kind="dock", n=48, rotations=1, t=1, batch=0, tile=0, lanes=0, entry="host"),
        # the command line's form: a default context docks the 360-rotation set with
        # host buffers in and out, three poses kept per rotation
        dict(name="default-128", kind="dock", n=128, rotations=360, t=3, batch=0, tile=0, lanes=0, entry="host"),
        # small-complex screening: the default 3,600-rotation set, best pose per rotation,
        # resident matrices and results
        dict(name="screen-96", kind="dock", n=96, rotations=3600, t=1, batch=192, tile=16, lanes=2, entry="device"),
        # the headline job's shape, 128^3 with three poses per rotation, from host buffers
        dict(name="headline-128", kind="dock", n=128, rotations=3600, t=3, batch=512, tile=16, lanes=1, entry="host"),
        # a grid edge whose half is odd (the padding does not prune evenly), and a long
        # pose list per rotation for later re-ranking
        dict(name="odd-126-t10", kind="dock", n=126, rotations=1200, t=10, batch=128, tile=16, lanes=2,
             entry="device"),
        # large single-domain receptors (4,000 residues size to about this grid)
        dict(name="large-160", kind="dock", n=160, rotations=1200, t=1, batch=128, tile=16, lanes=2, entry="device"),
        # multi-domain receptors: the largest grids whose planes stay in shared memory
        dict(name="large-216", kind="dock", n=216, rotations=360, t=3, batch=48, tile=16, lanes=2, entry="host"),
        # assemblies: planes pass through global memory
        dict(name="assembly-256", kind="dock", n=256, rotations=192, t=3, batch=32, tile=16, lanes=2, entry="device"),
        # the largest: an odd half edge above that, settings left as a fresh context has them
        # apart from the rotations per launch
        dict(name="assembly-330", kind="dock", n=330, rotations=64, t=1, batch=8, tile=32, lanes=2, entry="device"),
        # cross-docking: several pairs of uneven sizes through one graph
        dict(name="pairs-72-144", kind="pairs", sizes="72,84,96,108,120,144", rotations=480, t=1, batch=96, tile=16),
        # parameter fitting: the gradient of the smooth maximum over a rotation set's best poses
        dict(name="adjoint-96", kind="adjoint", n=96, rotations=3600, batch=64, temperature=10.0),
        # preparing a pair: receptor grids and spectrum from the atoms
        dict(name="receptor-128", kind="receptor", n=128),
    ]


def _built(lo, hi):
    return [n for n in range(lo, hi + 1, 2) if lib().md_fft_size_supported(n)]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above.  rng: random.Random."""
    what = rng.choice(("default", "batched", "batched", "batched", "pairs", "adjoint", "receptor"))
    if what == "receptor":
        return dict(kind="receptor", n=rng.choice(_built(48, 256)))
    if what == "adjoint":
        n = rng.choice(_built(48, 144))
        return dict(kind="adjoint", n=n, rotations=_logint(rng, 32, 3600), batch=rng.choice((16, 32, 64)),
                    temperature=rng.choice((5.0, 10.0, 20.0)))
    if what == "pairs":
        sizes = sorted(rng.choice(_built(60, 160)) for _ in range(rng.randint(2, 6)))
        top = int(min(600, 3e9 / sum(n ** 3 for n in sizes)))
        return dict(kind="pairs", sizes=",".join(map(str, sizes)), rotations=_logint(rng, 24, top),
                    t=rng.choice((1, 3)), batch=rng.choice((32, 64, 96)), tile=rng.choice((16, 32)))
    t = rng.choice((1, 1, 1, 3, 3, 5, 10, 20))
    if what == "default":
        n = rng.choice(_built(32, 168))
        top = int(min(360, 7.5e8 / n ** 3))
        return dict(kind="dock", n=n, rotations=_logint(rng, 1, top), t=t, batch=0, tile=0, lanes=0, entry="host")
    sizes = _built(48, 330)
    n = min(sizes, key=lambda v: abs(v - math.exp(rng.uniform(math.log(48), math.log(330)))))
    top = int(min(3600, (3.5e9 if n <= 160 and n % 4 == 0 else 1.4e9) / n ** 3))
    batch = min(_logint(rng, 4, 512), max(4, int(4e9 / (8.0 * n ** 3))))
    return dict(kind="dock", n=n, rotations=_logint(rng, min(16, top), top), t=t, batch=batch,
                tile=rng.choice((16, 16, 8, 32)), lanes=rng.choice((1, 2)), entry=rng.choice(("host", "device")))


# ------------------------------------------------------------------ inputs
def _rng(seed, *more):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, *more])


def _atoms(rng, semi, limit=None):
    """Random ellipsoid of atoms, semi-axis `semi` A along the longest axis;
    coordinates centred on the bounding box, radii and charges."""
    axes = semi * np.array([1.0, 0.8, 0.7])
    n = max(12, int(4.0 / 3.0 * math.pi * axes.prod() / ATOM_VOLUME))
    if limit and n > limit:
        axes *= (limit / n) ** (1.0 / 3.0)
        n = limit
    v = rng.normal(size=(n, 3))
    v *= (rng.random(n) ** (1.0 / 3.0) / np.linalg.norm(v, axis=1))[:, None]
    xyz = (v * axes).astype(np.float32)
    xyz -= ((xyz.max(0) + xyz.min(0)) / 2).astype(np.float32)
    return xyz, RADII[rng.integers(len(RADII), size=n)], CHARGES[rng.integers(len(CHARGES), size=n)]


def _receptor_atoms(n, seed):
    return _atoms(_rng(seed, n, 1), (GRID_WIDTH * (n // 2) - 16.0) / 2)


def _ligand_atoms(n, seed):
    return _atoms(_rng(seed, n, 2), 0.75 * (GRID_WIDTH * (n // 2) - 16.0) / 2, MAX_LIGAND_ATOMS)


def _rotations(count, seed):
    """ZXZ rotation matrices of random orientations, [count][9] float32."""
    rng = _rng(seed, count, 3)
    a, c = rng.uniform(0, 2 * math.pi, (2, count))
    b = np.arccos(rng.uniform(-1, 1, count))
    c0, s0, c1, s1, c2, s2 = np.cos(a), np.sin(a), np.cos(b), np.sin(b), np.cos(c), np.sin(c)
    m = np.stack([c0 * c2 - s0 * c1 * s2, -c0 * s2 - s0 * c1 * c2, s0 * s1,
                  s0 * c2 + c0 * c1 * s2, -s0 * s2 + c0 * c1 * c2, -c0 * s1,
                  s1 * s2, s1 * c2, c1], axis=1)
    return np.ascontiguousarray(m, dtype=np.float32)


def _grid_coord(ng):
    length = np.float32(GRID_WIDTH) * np.float32(ng)
    return (float(length) * (-0.5 + (0.5 + np.arange(ng)) / ng)).astype(np.float32)


def _receptor_grids(n, seed):
    """Receptor voxel grids as torch float32 on the GPU: core -45, outside it
    the number of atoms within reach of the surface shell, and the field of the
    charges (quantised, so that the sums do not depend on their order)."""
    ng = n // 2
    xyz, rad, q = _receptor_atoms(n, seed)
    dev = "cuda"
    x = torch.from_numpy(xyz).to(dev).double()
    r = torch.from_numpy(rad).to(dev).double()
    q = torch.from_numpy(q).to(dev).double()
    gc = torch.from_numpy(_grid_coord(ng)).to(dev).double()
    o = (x / GRID_WIDTH + ng // 2).long()
    core = torch.zeros(ng ** 3 + 1, dtype=torch.bool, device=dev)
    shell = torch.zeros(ng ** 3 + 1, dtype=torch.int32, device=dev)
    field = torch.zeros(ng ** 3 + 1, dtype=torch.int32, device=dev)
    span = torch.arange(-5, 6, device=dev)
    plane = torch.cartesian_prod(span, span)
    for di in range(-5, 6):
        c = o[:, None, :] + torch.cat([torch.full_like(plane[:, :1], di), plane], 1)[None]
        inside = ((c >= 0) & (c < ng)).all(-1)
        cc = c.clamp(0, ng - 1)
        d = ((x[:, None, :] - gc[cc]) ** 2).sum(-1)
        flat = torch.where(inside, (cc[..., 0] * ng + cc[..., 1]) * ng + cc[..., 2], ng ** 3)
        near = d < 1.5 * (r ** 2)[:, None]
        core[flat[near]] = True
        shell.index_add_(0, flat.reshape(-1), (d < ((r + 3.6) ** 2)[:, None]).int().reshape(-1))
        dist = d.sqrt().clamp(min=0.3)
        eps = torch.where(dist >= 8.0, 80.0, torch.where(dist > 6.0, 38.0 * dist - 224.0, 4.0))
        term = (-2800.0 * q[:, None] / eps / dist * 64.0).round().int()
        field.index_add_(0, flat.reshape(-1), term.reshape(-1))
    core, shell, field = core[:-1], shell[:-1], field[:-1]
    real = torch.where(core, -45.0, shell.float())
    imag = torch.where(core, 0.0, field.float() / 64.0)
    return real.reshape(ng, ng, ng), imag.reshape(ng, ng, ng)


def _context(n, seed, stream=None):
    """A context prepared for one pair: grid, receptor, ligand."""
    fp = FFTProcess(0, stream=stream)
    fp.alloc_array(n, GRID_WIDTH, _grid_coord(n // 2))
    real, imag = _receptor_grids(n, seed)
    fp.receptor_fft(real.cpu().numpy(), imag.cpu().numpy())
    fp.ligand_data_transfer_gpu(*_ligand_atoms(n, seed))
    return fp


def _pose_out(count):
    return torch.zeros(count * 5, dtype=torch.int32, device="cuda")


def _pose_views(out):
    """Scores and (rotation, i, j, k) of a device pose buffer."""
    rec = out.view(-1, 5)
    return {"score": rec.view(torch.float32)[:, 0], "cell": rec[:, 1:]}


def _adjoint_inputs(case, seed):
    """Rotation matrices and best-pose records with the spread of a docking
    run's best scores; translations bring the ligand into contact."""
    n, count = case["n"], case["rotations"]
    rng = _rng(seed, n, count, 4)
    top = np.zeros(count, POSE_DTYPE)
    score = rng.normal(1500.0, 475.0, count)
    near = np.quantile(score, 0.995) if count > 1 else score[0]      # the orientations around the best pose score alike
    score = np.where(score >= near, near + rng.normal(0.0, 8.0, count), score)
    top["score"] = np.maximum(1.0, score)
    top["rot"] = np.arange(count)
    u = rng.normal(size=(count, 3))
    u *= (rng.uniform(0.25, 0.42, count) * (n // 2) / np.linalg.norm(u, axis=1))[:, None]
    t = np.round(u).astype(np.int64) % n
    top["i"], top["j"], top["k"] = t[:, 0], t[:, 1], t[:, 2]
    return _rotations(count, seed), top


def prepare(case, seed):
    if case["kind"] == "dock":
        stream = torch.cuda.Stream() if case["entry"] == "device" else None
        fp = _context(case["n"], seed, stream.cuda_stream if stream else None)
        if case["batch"]:
            fp.set_batch(case["batch"])
            fp.set_tile(case["tile"])
            fp.set_lanes(case["lanes"])
        mats = _rotations(case["rotations"], seed)
        if stream is None:
            return dict(case=case, fp=fp, mats=mats)
        return dict(case=case, fp=fp, stream=stream, mats=torch.from_numpy(mats).cuda(),
                    out=_pose_out(case["rotations"] * case["t"]))
    if case["kind"] == "pairs":
        stream = torch.cuda.Stream()
        sizes = [int(v) for v in case["sizes"].split(",")]
        ctxs = []
        for p, n in enumerate(sizes):
            fp = _context(n, seed + 1000 * p)
            fp.set_batch(case["batch"])
            fp.set_tile(case["tile"])
            ctxs.append(fp)
        mats = torch.from_numpy(_rotations(case["rotations"], seed)).cuda()
        outs = [_pose_out(case["rotations"] * case["t"]) for _ in ctxs]
        k = len(ctxs)
        args = ((C.c_void_p * k)(*[fp._h.value for fp in ctxs]), k, (C.c_void_p * k)(*[mats.data_ptr()] * k),
                (C.c_int * k)(*[case["rotations"]] * k), case["t"], (C.c_void_p * k)(*[o.data_ptr() for o in outs]))
        return dict(case=case, ctxs=ctxs, runner=FFTProcess(0, stream=stream.cuda_stream), stream=stream, mats=mats,
                    outs=outs, args=args)
    if case["kind"] == "adjoint":
        fp = _context(case["n"], seed)
        fp.set_batch(case["batch"])
        mats, top = _adjoint_inputs(case, seed)
        return dict(case=case, fp=fp, mats=mats, top=top)
    fp = FFTProcess(0)
    fp.alloc_array(case["n"], GRID_WIDTH, _grid_coord(case["n"] // 2))
    xyz, rad, q = _receptor_atoms(case["n"], seed)
    ace = _rng(seed, case["n"], 5).uniform(-1.2, 1.2, len(rad)).astype(np.float32)
    return dict(case=case, fp=fp, atoms=(xyz, rad, q, ace))


def run(state):
    case = state["case"]
    if case["kind"] == "dock" and case["entry"] == "host":
        poses = state["fp"].cuda_fft(state["mats"], t=case["t"])
        cell = np.stack([poses["rot"], poses["i"], poses["j"], poses["k"]], axis=1)
        return {"score": poses["score"].copy(), "cell": cell}
    if case["kind"] == "dock":
        stream = state["stream"]
        stream.wait_stream(torch.cuda.current_stream())
        state["fp"].dock_device(state["mats"].data_ptr(), 0, case["rotations"], case["t"], state["out"].data_ptr())
        torch.cuda.current_stream().wait_stream(stream)
        return _pose_views(state["out"])
    if case["kind"] == "pairs":
        stream = state["stream"]
        stream.wait_stream(torch.cuda.current_stream())
        rc = lib().md_dock_pairs(state["runner"]._h, *state["args"])
        if rc:
            raise RuntimeError(lib().md_last_error(state["runner"]._h).decode())
        torch.cuda.current_stream().wait_stream(stream)
        return [_pose_views(o) for o in state["outs"]]
    if case["kind"] == "adjoint":
        g = state["fp"].adjoint_lse(state["mats"], state["top"], temperature=case["temperature"], alpha=1.0)
        return {k: g[k] for k in ("loss", "d_rec_r", "d_rec_i", "d_charge", "d_alpha")}
    real, imag = state["fp"].receptor_build(*state["atoms"], return_grids=True)
    return {"real": real, "imag": imag}


# ------------------------------------------------------------------ what a pass cannot do without
def _dock_flops(n):
    """Real operations of one rotation's transforms: pruned forward complex
    FFT (z on a quarter of the lines, y on half, x on all), the product with
    the conjugate spectrum, and the inverse of the Hermitian half."""
    return 3.25 * n * n * 5.0 * n * math.log2(n) + 12.0 * n ** 3


def work(case):
    if case["kind"] == "dock":
        n, r = case["n"], case["rotations"]
        return {"bytes": 8.0 * n ** 3 + 24.0 * len(_ligand_atoms(n, 0)[1]) + r * (36.0 + 20.0 * case["t"]),
                "flops": r * _dock_flops(n)}
    if case["kind"] == "pairs":
        sizes = [int(v) for v in case["sizes"].split(",")]
        r = case["rotations"]
        return {"bytes": sum(8.0 * n ** 3 + r * (36.0 + 20.0 * case["t"]) for n in sizes),
                "flops": sum(r * _dock_flops(n) for n in sizes)}
    ng3 = float((case["n"] // 2) ** 3)
    if case["kind"] == "adjoint":
        # every weighted rotation's ligand cells added into the receptor gradient once
        cells = len(_ligand_atoms(case["n"], 0)[1]) * 10.0
        return {"bytes": 16.0 * ng3 + 56.0 * case["rotations"], "flops": 2.0 * cells * case["rotations"]}
    # receptor: every atom's shell and field cells, then the forward transform
    n = case["n"]
    atoms = len(_receptor_atoms(n, 0)[1])
    return {"bytes": 28.0 * atoms + 8.0 * ng3 + 8.0 * n ** 3,
            "flops": atoms * (1331.0 * 10 + 1331.0 * 12) + 1.75 * n * n * 5.0 * n * math.log2(n)}


def tolerance(case):
    if case["kind"] == "receptor":
        return "exact"                  # the grids are MEGADOCK's floats bit for bit
    if case["kind"] == "adjoint":
        return {"rel": 4e-7}            # four times the largest error against exact (7e-8 to 1e-7)
    # 32-bit transforms of grids whose largest correlations (-45 x core cells)
    # are many times the best scores, the more the larger the grid: four times
    # the errors against exact (up to 1e-5 at 160, 4e-5 at 330).  Poses of a
    # list swap where two scores tie to rounding (0.3 % of the whole numbers
    # seen; a swap is up to eight of them).
    count = case["rotations"] * case["t"] * 4
    large = max(int(v) for v in case["sizes"].split(",")) if case["kind"] == "pairs" else case["n"]
    tol = {"rel": 4e-5, "max": 1.6e-4} if large <= 168 else {"rel": 1.6e-4, "max": 5.3e-4}
    return dict(tol, differ=min(0.5, max(1.2e-2, 16.0 / count)))


# ------------------------------------------------------------------ 64-bit answers
def _voxels(n, mats, xyz, rad, q):
    """Ligand grids of a chunk of rotations: occupancy (every cell of a
    surviving core cell or a surface cell is 1) and charge sums, float64.
    The cell decisions are float32 comparisons by definition."""
    ng = n // 2
    count = len(mats)
    dev = "cuda"
    gw = torch.tensor(GRID_WIDTH, dtype=torch.float32, device=dev)
    gc = torch.from_numpy(_grid_coord(ng)).to(dev)
    a = [torch.from_numpy(np.ascontiguousarray(xyz[:, d])).to(dev)[None] for d in range(3)]
    m = torch.from_numpy(mats).to(dev)[:, :, None]
    pos = [(m[:, 3 * d] * a[0] + m[:, 3 * d + 1] * a[1]) + m[:, 3 * d + 2] * a[2] for d in range(3)]
    r2 = torch.from_numpy(rad).to(dev)
    r2 = r2 * r2
    core = torch.zeros(count * ng ** 3 + 1, dtype=torch.bool, device=dev)
    surf = torch.zeros(count * ng ** 3 + 1, dtype=torch.bool, device=dev)
    base = torch.arange(count, device=dev)[:, None] * ng ** 3
    org = [torch.trunc(p / gw + float(ng // 2)).long() for p in pos]
    sq, idx = [], []
    for d in range(3):
        rows, ids = [], []
        for o in range(-2, 3):
            i = org[d] + o
            ok = (i >= 0) & (i < ng)
            diff = pos[d] - gc[i.clamp(0, ng - 1)]
            rows.append(torch.where(ok, diff * diff, torch.inf))
            ids.append(i.clamp(0, ng - 1))
        sq.append(rows)
        idx.append(ids)
    for oi in range(5):
        for oj in range(5):
            dxy = sq[0][oi] + sq[1][oj]
            for ok_ in range(5):
                d3 = dxy + sq[2][ok_]
                flat = base + (idx[0][oi] * ng + idx[1][oj]) * ng + idx[2][ok_]
                core[torch.where(d3 < r2 * 1.5, flat, count * ng ** 3).reshape(-1)] = True
                surf[torch.where(d3 < r2, flat, count * ng ** 3).reshape(-1)] = True
    core = core[:-1].view(count, ng, ng, ng)
    surf = surf[:-1].view(count, ng, ng, ng)
    inner = core.clone()
    for axis in (1, 2, 3):
        for step in (1, -1):
            inner &= torch.roll(core, step, axis)
    keep = core.clone()
    keep[:, 1:-1, 1:-1, 1:-1] &= inner[:, 1:-1, 1:-1, 1:-1]
    occ = (keep | surf).double()
    pad = torch.tensor(np.float32(ng * np.float32(GRID_WIDTH)) / np.float32(2), dtype=torch.float32, device=dev)
    cell = [torch.trunc((p + pad) / gw).long().clamp(0, ng - 1) for p in pos]
    flat = base + (cell[0] * ng + cell[1]) * ng + cell[2]
    chg = torch.zeros(count * ng ** 3, dtype=torch.float64, device=dev)
    chg.index_add_(0, flat.reshape(-1), torch.from_numpy(q).to(dev).double().repeat(count))
    return occ, chg.view(count, ng, ng, ng), cell


def _embed(n, real, imag):
    ng, off = n // 2, n // 4
    g = torch.zeros(real.shape[:-3] + (n, n, n), dtype=torch.complex128, device="cuda")
    g[..., off:off + ng, off:off + ng, off:off + ng] = torch.complex(real.double(), imag.double())
    return g


def _exact_dock(n, seed, rotations, t, mats):
    spec = torch.fft.fftn(_embed(n, *_receptor_grids(n, seed))).conj()
    lig = _ligand_atoms(n, seed)
    chunk = max(1, min(16, int(4e6 / n ** 2 / 10), int(2e9 / (16 * n ** 3))))
    score, cell = [], []
    for r0 in range(0, rotations, chunk):
        occ, chg, _ = _voxels(n, mats[r0:r0 + chunk], *lig)
        g = torch.fft.fftn(_embed(n, occ, chg), dim=(-3, -2, -1)) * spec
        s = torch.fft.ifftn(g, dim=(-3, -2, -1)).real.reshape(len(occ), -1)
        top, at = torch.topk(s, t, dim=1)
        if t == 1:
            at = torch.where(top > 0, at, torch.zeros_like(at))
            top = top.clamp(min=0.0)
        rot = (r0 + torch.arange(len(occ), device="cuda"))[:, None].expand_as(at)
        cell.append(torch.stack([rot, at // (n * n), at // n % n, at % n], -1).reshape(-1, 4))
        score.append(top.reshape(-1))
    return {"score": torch.cat(score).cpu().numpy(), "cell": torch.cat(cell).cpu().numpy()}


def _exact_adjoint(case, seed):
    n, ng, off = case["n"], case["n"] // 2, case["n"] // 4
    mats, top = _adjoint_inputs(case, seed)
    lig = _ligand_atoms(n, seed)
    real, imag = _receptor_grids(n, seed)
    s = top["score"].astype(np.float64)
    e = np.exp((s - s.max()) / case["temperature"])
    w = e / e.sum()
    loss = s.max() + case["temperature"] * math.log(e.sum())
    drr = torch.zeros(ng, ng, ng, dtype=torch.float64, device="cuda")
    dri = torch.zeros_like(drr)
    dq = torch.zeros(len(lig[1]), dtype=torch.float64, device="cuda")
    zi = torch.zeros(n, n, n, dtype=torch.float64, device="cuda")
    zi[off:off + ng, off:off + ng, off:off + ng] = imag.double()
    here = torch.arange(ng, device="cuda") + off
    live = np.flatnonzero(w > 1e-30)
    for r0 in range(0, len(live), 8):
        part = live[r0:r0 + 8]
        occ, chg, cell = _voxels(n, mats[part], *lig)
        both = _embed(n, occ, chg)
        for m, r in enumerate(part):
            t = [int(top[a][r]) for a in "ijk"]
            at = [(here + v) % n for v in t]
            g = both[m][at[0][:, None, None], at[1][None, :, None], at[2][None, None, :]]
            drr += w[r] * g.real
            dri += w[r] * g.imag
            c = [(cell[d][m] + off - t[d]) % n for d in range(3)]
            dq += w[r] * zi[c[0], c[1], c[2]]
    return {"loss": loss, "d_rec_r": drr.cpu().numpy(), "d_rec_i": dri.cpu().numpy(), "d_charge": dq.cpu().numpy(),
            "d_alpha": float((dri * imag.double()).sum())}


def exact(case, seed):
    if case["kind"] == "receptor":
        # the open-space marking sweeps the cells one after another in place: minutes in numpy
        return None
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    if case["kind"] == "pairs":
        mats = _rotations(case["rotations"], seed)
        return [_exact_dock(int(v), seed + 1000 * p, case["rotations"], case["t"], mats)
                for p, v in enumerate(case["sizes"].split(","))]
    return _exact_dock(case["n"], seed, case["rotations"], case["t"], _rotations(case["rotations"], seed))
