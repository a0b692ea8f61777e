"""Performance cases: what a user of the framework has it do, over the range of sizes,
types and directions that its layers serve.

``listed()`` names the cases, ``draw(rng)`` gives others of the same ranges,
``prepare`` makes a case's inputs on the GPU from a seed, ``run`` is one pass through
the public layers, ``work`` the bytes and operations a pass cannot do without, and
``exact`` the result in 64 bits from plain torch.

A case is a dict: ``kind`` (below), ``dtype``, ``batch``, ``lo`` and ``hi`` (shortest and
longest chain: residues, or atoms for the kinds that start from coordinates; the rows
are padded to ``hi``, as a data loader pads to its longest chain), ``grad`` (forward
and backward, or forward alone) and ``graph`` (the pass is captured once in a CUDA
graph by the program and replayed, or called eagerly).

  backbone   Angles2Backbone
  fullatom   Angles2Coords, names included
  train      Angles2Coords -> Coords2RMSD -> mean -> dL/dangles
  typed      Coords2TypedCoords and its backward
  score      Coords2RMSD of decoys against targets
  pose       Coords2Center, CoordsTranslate, CoordsRotate, getBBox and the backward
"""
import math

import numpy as np
import torch

ATOMS_PER_RESIDUE = 8.35  # heavy atoms per residue of a uniformly random sequence
LETTERS = "GASCVILTRKDNEQMHPFYW"


def listed():
    return [
        # a gradient check or the first steps with the library: 32 peptides of 64 residues, one
        # call forward and one backward, where latency and host time count
        dict(name="backbone_small", kind="backbone", dtype="float32", batch=32, lo=64, hi=64, grad=True, graph=False),
        # the double-precision layer on a batch of small domains (reference values, gradient checks)
        dict(name="backbone_f64", kind="backbone", dtype="float64", batch=256, lo=60, hi=350, grad=True, graph=False),
        # one training batch of mixed proteins, forward and backward replayed as one CUDA graph
        dict(name="backbone_ragged", kind="backbone", dtype="float32", batch=1024, lo=20, hi=700, grad=True, graph=True),
        # the same at a padded length that is not a multiple of four, as the longest chain of a batch usually is
        dict(name="backbone_odd", kind="backbone", dtype="float32", batch=2048, lo=100, hi=517, grad=True, graph=True),
        # the large throughput sweep: 4096 chains of 1000 residues
        dict(name="backbone_large", kind="backbone", dtype="float32", batch=4096, lo=1000, hi=1000, grad=True, graph=True),
        # building a handful of full-atom structures from predicted angles: forward only, latency
        dict(name="fullatom_small", kind="fullatom", dtype="float32", batch=8, lo=90, hi=251, grad=False, graph=False),
        # double precision full-atom batch, forward and backward
        dict(name="fullatom_f64", kind="fullatom", dtype="float64", batch=64, lo=150, hi=150, grad=True, graph=False),
        # large full-atom batch: coordinates and names, then dL/dangles
        dict(name="fullatom_large", kind="fullatom", dtype="float32", batch=4096, lo=500, hi=500, grad=True, graph=False),
        # the training step: full-atom chains against target structures, RMSD loss, one CUDA graph
        dict(name="train_step", kind="train", dtype="float32", batch=256, lo=50, hi=500, grad=True, graph=True),
        # atoms regrouped by type for a volumetric network, with the gradient's way back
        dict(name="typed", kind="typed", dtype="float32", batch=4096, lo=50, hi=500, grad=True, graph=False),
        # scoring a set of decoys against their targets: forward only
        dict(name="score", kind="score", dtype="float32", batch=4096, lo=400, hi=2303, grad=False, graph=False),
        # random poses of a batch of structures (data augmentation), differentiable
        dict(name="pose", kind="pose", dtype="float32", batch=4096, lo=1000, hi=3471, grad=True, graph=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["backbone", "backbone", "backbone", "fullatom", "fullatom", "train", "typed", "score", "pose"])
    f64 = kind in ("backbone", "fullatom") and rng.random() < 0.25
    # (batch range, length range, most batch * length)
    ranges = {
        "backbone": ((8, 256), (30, 500), 89600) if f64 else ((16, 4096), (30, 1000), 4096000),
        "fullatom": ((4, 64), (20, 300), 9600) if f64 else ((1, 4096), (20, 500), 2048000),
        "train": ((16, 512), (50, 500), 128000),
        "typed": ((64, 4096), (50, 500), 2048000),
        "score": ((64, 4096), (200, 4000), 9433088),
        "pose": ((64, 4096), (200, 4000), 14217216),
    }
    (b0, b1), (l0, l1), most = ranges[kind]
    while True:
        batch, hi = _log_int(rng, b0, b1), _log_int(rng, l0, l1)
        if batch * hi <= most:
            break
    lo = hi if rng.random() < 0.25 else max(l0 // 2, int(hi * rng.uniform(0.05, 0.9)))
    grad = kind in ("train", "typed", "pose", "backbone") or (kind == "fullatom" and rng.random() < 0.7)
    graph = kind == "train" or (kind == "backbone" and not f64 and rng.random() < 0.7)
    return dict(kind=kind, dtype="float64" if f64 else "float32", batch=batch, lo=lo, hi=hi, grad=grad, graph=graph)


# ------------------------------------------------------------------ inputs
def _lengths(case, rng):
    n = rng.integers(case["lo"], case["hi"] + 1, case["batch"])
    n[int(rng.integers(case["batch"]))] = case["hi"]
    return n.astype(np.int32)


def _sequences(n, L, rng):
    """Uniformly random residue letters [B, L].  One of the longest chains is rich in
    large residues, with an atom count that depends on L alone (the random ones stay
    below it), so that the padded atom count of a batch does not change with the seed."""
    letters = np.frombuffer(LETTERS.encode(), dtype=np.uint8)[rng.integers(0, 20, (len(n), L))]
    row = np.arange(L) % 20
    order = np.argsort(_NATOMS[row], kind="stable")
    most = min(14 * L, 8.35 * L + 13.0 * math.sqrt(L))
    for k in order:
        if _NATOMS[row].sum() >= most:
            break
        row[k] = 19
    letters[int(np.argmax(n))] = np.frombuffer(LETTERS.encode(), dtype=np.uint8)[rng.permutation(row)]
    return letters


def _inputs(case, seed):
    """Plain tensors on the GPU (and sequences), from the seed alone."""
    dev = torch.device("cuda")
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=dev).manual_seed(int(rng.integers(1 << 31)))
    dt = getattr(torch, case["dtype"])
    B, L, kind = case["batch"], case["hi"], case["kind"]
    n = _lengths(case, rng)
    lengths = torch.from_numpy(n).to(dev)
    real = torch.arange(L, device=dev)[None, :] < lengths[:, None]

    def uniform(*shape):
        return (torch.rand(*shape, dtype=dt, device=dev, generator=gen) * 2 - 1) * math.pi

    def normal(*shape):
        return torch.randn(*shape, dtype=dt, device=dev, generator=gen)

    if kind in ("backbone", "fullatom", "train"):
        rows = 3 if kind == "backbone" else 8
        ang = uniform(B, rows, L)
        ang[:, 2] = math.pi + 0.05 * normal(B, L)
        ang *= real[:, None, :]
        out = dict(angles=ang, lengths=lengths)
        if kind == "backbone":
            out["up"] = normal(B, 9 * L)
            return out
    if kind in ("fullatom", "train", "typed"):
        letters = _sequences(n, L, rng)
        seqs = [bytes(row[:k]).decode() for row, k in zip(letters, n)]
        types = np.where(np.arange(L)[None, :] < n[:, None], _TYPE_OF_BYTE[letters], 20)
        counts = _NATOMS[types].sum(1)
        max_atoms = int(counts.max())
        if kind == "typed":
            return dict(seqs=seqs, coords=15.0 * normal(B, 3 * max_atoms), up=normal(B, 3 * max_atoms))
        out.update(seqs=seqs, types=torch.from_numpy(types).to(dev), max_atoms=max_atoms)
        if kind == "fullatom":
            out["up"] = normal(B, 3 * max_atoms)
        else:  # targets: the structures of perturbed angles
            noisy = (ang + 0.3 * normal(B, 8, L)) * real[:, None, :]
            with torch.no_grad():
                out["target"] = _full_atom(noisy.double(), out["types"], max_atoms).to(dt)
            out["num_atoms"] = torch.from_numpy(counts.astype(np.int32)).to(dev)
        return out
    # coordinates of compact chains: a random walk drawn towards its own mean
    x = normal(B, L, 3).cumsum(1) * 1.5
    x = (x - x.mean(1, keepdim=True)) * 0.6 + 10.0 * normal(B, 1, 3)
    x = (x * real[..., None]).reshape(B, 3 * L)
    q = torch.randn(B, 4, dtype=torch.float64, device=dev, generator=gen)
    w, i, j, k = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    rot = torch.stack([w * w + i * i - j * j - k * k, 2 * (i * j - w * k), 2 * (i * k + w * j),
                       2 * (i * j + w * k), w * w - i * i + j * j - k * k, 2 * (j * k - w * i),
                       2 * (i * k - w * j), 2 * (j * k + w * i), w * w - i * i - j * j + k * k], 1).view(B, 3, 3)
    out = dict(coords=x, num_atoms=lengths, real=real)
    if kind == "score":
        y = (x.view(B, L, 3).double() @ rot.transpose(1, 2)).to(dt) + 2.0 * normal(B, L, 3)
        out["target"] = (y * real[..., None]).reshape(B, 3 * L)
    else:
        out.update(rot=rot.to(dt), up=normal(B, 3 * L))
    return out


# ------------------------------------------------------------------ one pass
def _pass(state):
    kind, s = state["case"]["kind"], state["in"]
    if kind == "backbone":
        coords = state["layer"](state["angles"], s["lengths"])
        if not state["case"]["grad"]:
            return [coords]
        grad, = torch.autograd.grad(coords, state["angles"], s["up"])
        return [coords.detach(), grad]
    if kind == "fullatom":
        coords, res, atom, num = state["layer"](state["angles"], s["seqs"])
        if not state["case"]["grad"]:
            return [coords, res, atom, num]
        grad, = torch.autograd.grad(coords, state["angles"], s["up"])
        return [coords.detach(), res, atom, num, grad]
    if kind == "train":
        coords = state["layer"](state["angles"], s["seqs"])[0]
        rmsd = state["rmsd"](coords, s["target"], s["num_atoms"])
        grad, = torch.autograd.grad(rmsd.mean(), state["angles"])
        return [rmsd.detach(), grad]
    if kind == "typed":
        out, n, off = state["layer"](state["coords"], state["res"], state["atom"], state["num"])
        grad, = torch.autograd.grad(out, state["coords"], s["up"])
        return [out.detach(), n, off, grad]
    if kind == "score":
        return [state["rmsd"](s["coords"], s["target"], s["num_atoms"]), state["rmsd"].UT]
    center = state["center"](s["coords"], s["num_atoms"])
    moved = state["translate"](state["coords"], -center, s["num_atoms"])
    turned = state["rotate"](moved, s["rot"], s["num_atoms"])
    lo, hi = state["bbox"](turned.detach(), s["num_atoms"])
    grad, = torch.autograd.grad(turned, state["coords"], s["up"])
    return [center, turned.detach(), lo, hi, grad]


def prepare(case, seed):
    from torchproteinlibrary_gb300.FullAtomModel import Angles2Coords, Coords2TypedCoords
    from torchproteinlibrary_gb300.FullAtomModel.CoordsTransform import (Coords2Center, CoordsRotate, CoordsTranslate,
                                                                         getBBox)
    from torchproteinlibrary_gb300.ReducedModel import Angles2Backbone
    from torchproteinlibrary_gb300.RMSD import Coords2RMSD

    s = _inputs(case, seed)
    state = {"case": case, "in": s}
    kind = case["kind"]
    if "angles" in s:
        state["angles"] = s["angles"].clone().requires_grad_(case["grad"])
    if kind == "backbone":
        state["layer"] = Angles2Backbone()
    elif kind in ("fullatom", "train"):
        state["layer"] = Angles2Coords()
    elif kind == "typed":
        with torch.no_grad():  # the names and counts that go with the sequences
            zero = torch.zeros(case["batch"], 8, case["hi"], device="cuda")
            _, state["res"], state["atom"], state["num"] = Angles2Coords()(zero, s["seqs"])
        state["layer"] = Coords2TypedCoords()
        state["coords"] = s["coords"].clone().requires_grad_()
    elif kind == "pose":
        state.update(center=Coords2Center(), translate=CoordsTranslate(), rotate=CoordsRotate(), bbox=getBBox,
                     coords=s["coords"].clone().requires_grad_())
    if kind in ("train", "score"):
        state["rmsd"] = Coords2RMSD()
    if case["graph"]:  # the program's own capture of the pass, as torch.cuda.graph asks: warmed up on a side stream
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                _pass(state)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            state["out"] = _pass(state)
        state["graph"] = graph
    return state


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    return _pass(state)


def work(case):
    B, L, size = case["batch"], case["hi"], 8 if case["dtype"] == "float64" else 4
    n = 0.5 * (case["lo"] + case["hi"]) * B  # residues, or atoms where coordinates come in
    kind, back = case["kind"], 1 if case["grad"] else 0
    if kind == "backbone":  # angles in, coordinates out; dL/dx in, dL/dangles out
        return {"bytes": size * (3 * n + 9 * B * L + back * (9 * n + 3 * B * L)), "flops": n * (400 + back * 250)}
    atoms = ATOMS_PER_RESIDUE
    if kind in ("fullatom", "train"):
        fwd = size * (8 * n + 3 * atoms * n) + n
        if kind == "fullatom":  # coordinates and two name words per atom out; dL/dx in, dL/dangles out
            return {"bytes": fwd + 8 * atoms * n + back * size * (3 * atoms * n + 8 * B * L),
                    "flops": n * (900 + back * 600)}
        # angles, sequence and target in, dL/dangles out: nothing between has to leave the chip
        return {"bytes": size * (8 * n + 3 * atoms * n + 8 * B * L) + n, "flops": n * (1500 + 60 * atoms)}
    if kind == "typed":  # coordinates and names in, coordinates out; dL/dtyped in, dL/dx out
        rows = atoms * B * L
        return {"bytes": atoms * n * (3 * size + 8) + 3 * size * rows + 3 * size * (atoms * n + rows),
                "flops": 10 * atoms * n}
    if kind == "score":
        return {"bytes": 6 * size * n, "flops": 36 * n}
    # coordinates in, posed coordinates out; dL/dx in, dL/dx out
    return {"bytes": size * (6 * n + 6 * B * L), "flops": 45 * n}


# ------------------------------------------------------------------ 64-bit results in plain torch
# Geometry of the kinematic chain: a joint is Ry(beta) Tx(d) Rx(alpha).  Per residue
# type the side-chain joints (beta, d, atoms in the joint's frame; joint k turns by chi
# k, Ala's by none) below the fixed rotation DUMMY about the N-CA bond's frame.
_H = 0.5 * math.pi
_RAD = math.pi / 180.0
_BB = ((math.pi - 1.9391, 1.460), (math.pi - 2.061, 1.525), (math.pi - 2.1186, 1.330))
_DUMMY = _H * 122.6860 / 180.0
_TETRA = -(math.pi - math.pi * 109.5 / 180.0)
_CO = (1.417 * math.cos(math.pi - 2.1033), 0.0, 1.417 * math.sin(math.pi - 2.1033))
_PRO = ((0.36842372, -1.29540981, 0.70468246), (-0.76137817, -2.21546205, 0.39299099),
        (-1.97838492, -1.33927458, 0.35849352))


def _bent(r, angle, side):  # a bond of length r in the x-z plane at `angle` from the incoming bond
    return (r * math.sin(angle - _H), 0.0, side * r * math.cos(angle - _H))


def _polar(r, angle):
    return (r * math.cos(angle), r * math.sin(angle), 0.0)


def _tilted(r, incline, turn, side):  # a bond inclined from x, turned about it
    c, s = math.cos(incline - _H), math.sin(incline - _H)
    return (r * s, side * r * c * math.sin(turn), r * c * math.cos(turn))


def _side_chains():
    o, cb, cc = (0.0, 0.0, 0.0), (_TETRA, 1.52), 1.527
    xz = lambda r, a: (r * math.cos(a), 0.0, r * math.sin(a))  # noqa: E731
    first, g = 110.7 * _RAD, 1.88444687881
    ring = [(0.69229424, -1.20533343, 0.0), (2.08228309, -1.20846014, 0.0), (2.77997771, -0.00625341, 0.0),
            (2.08768347, 1.19908002, 0.0), (0.69769462, 1.20220673, 0.0)]
    plain, two = (*cb, [o]), lambda r1, a1, r2, a2: [o, _bent(r1, a1, 1), _bent(r2, a2, -1)]  # noqa: E731
    acid, amide = two(1.25, 119.22 * _RAD, 1.25, 119.22 * _RAD), two(1.23, 120.85 * _RAD, 1.33, 116.48 * _RAD)
    bend = lambda deg: -(math.pi - math.pi * deg / 180.0)  # noqa: E731
    t = 1.90291866134 / 2
    return {
        "G": [], "P": [], "A": [plain],
        "S": [(*cb, [o, xz(1.417, -(math.pi - 110.773 * _RAD))])],
        "C": [(*cb, [o, xz(1.808, -(math.pi - 113.8169 * _RAD))])],
        "V": [(*cb, [o, _tilted(cc, first, g / 2, 1), _tilted(cc, first, g / 2, -1)])],
        "I": [(*cb, [o, _tilted(cc, first, g, 1)]),
              (*cb, [o, (1.52 * math.cos(math.pi - 113.97 * _RAD), 0.0, -1.52 * math.sin(math.pi - 113.97 * _RAD))])],
        "L": [plain, (*cb, [o, _tilted(cc, first, g / 2, 1), _tilted(cc, first, g / 2, -1)])],
        "T": [(*cb, [o, _tilted(1.417, 109.18 * _RAD, t, 1), _tilted(cc, first, t, -1)])],
        "R": [plain, plain, plain, (bend(111.68), 1.46, [o]), (bend(124.79), 1.33, two(1.33, 124.79 * _RAD, 1.33, 124.79 * _RAD))],
        "K": [plain, plain, plain, (_TETRA, 1.46, [o]), (bend(124.79), 1.33, [o])],
        "D": [plain, (*cb, acid)], "N": [plain, (*cb, amide)],
        "E": [plain, plain, (*cb, acid)], "Q": [plain, plain, (*cb, amide)],
        "M": [plain, plain, (bend(112.69), 1.81, [o]), (bend(100.61), 1.79, [o])],
        "H": [plain, (*cb, [o, _polar(1.35, -(math.pi - 2.27957453603)), _polar(2.1912, -(math.pi - 2.90352974362)),
                            _polar(2.1915, math.pi - 2.75209584734), _polar(1.38, math.pi - 2.14413698608)])],
        "F": [plain, (*cb, [o] + ring)], "Y": [plain, (*cb, [o] + ring + [(4.16960749, 0.05377697, 0.0)])],
        "W": [plain, (*cb, [o, (0.829890578, -1.09003744, 0.0), (0.84949676, 1.15028973, 0.0),
                            (2.1363699, -0.64570528, 0.0), (2.18136443, 0.71889842, 0.0), (0.61303306, 2.5301684, 0.0),
                            (3.22086556, 1.65663275, 0.0), (1.68979906, 3.42486545, 0.0), (2.92849902, 3.0257584, 0.0)])],
    }


_SIDE = _side_chains()
_NATOMS = np.array([7 if c == "P" else 4 + sum(len(j[2]) for j in _SIDE[c]) for c in LETTERS] + [0])  # 20: padding
_TYPE_OF_BYTE = np.full(256, 20)
_TYPE_OF_BYTE[np.frombuffer(LETTERS.encode(), dtype=np.uint8)] = np.arange(20)


def _turn(alpha, cb, sb):
    """Rotations Ry(beta) Rx(alpha), [..., 3, 3]."""
    ca, sa = torch.cos(alpha), torch.sin(alpha)
    zero = torch.zeros_like(ca)
    return torch.stack([cb + zero, sb * sa, sb * ca, zero, ca, -sa, zero - sb, cb * sa, cb * ca], -1).reshape(
        *alpha.shape, 3, 3)


def _backbone_frames(phi_psi_omega):
    """Rotations [B, 3L + 1, 3, 3] and positions [B, 3L + 1, 3] along N, CA, C, N, ..., C, N."""
    a = phi_psi_omega
    B, _, L = a.shape
    turns = torch.stack([_turn(a[:, k], math.cos(_BB[k][0]), math.sin(_BB[k][0])) for k in range(3)], 2)
    R = torch.eye(3, dtype=a.dtype, device=a.device).expand(B, 3, 3)
    all_r = [R]
    for m in turns.reshape(B, 3 * L, 3, 3).unbind(1):
        R = R @ m
        all_r.append(R)
    R = torch.stack(all_r, 1)
    bond = torch.tensor([[d * math.cos(b), 0.0, -d * math.sin(b)] for b, d in _BB], dtype=a.dtype, device=a.device)
    step = (R[:, :-1] @ bond.repeat(L, 1)[None, :, :, None]).squeeze(-1)
    return R, torch.cat([torch.zeros_like(step[:, :1]), step.cumsum(1)], 1)


def _backbone(ang, lengths):
    B, _, L = ang.shape
    _, p = _backbone_frames(ang)
    keep = torch.arange(L, device=ang.device)[None, :] < lengths[:, None]
    return (p[:, :-1].reshape(B, L, 9) * keep[..., None]).reshape(B, 9 * L)


def _full_atom(ang, types, max_atoms):
    """Heavy atoms [B, 3 max_atoms] of angles [B, 8, L] and residue types [B, L] (20: padding)."""
    dev, dt = ang.device, ang.dtype
    B, _, L = ang.shape
    R, p = _backbone_frames(ang[:, :3])
    R, p = R[:, :-1].reshape(B, L, 3, 3, 3), p[:, :-1].reshape(B, L, 3, 3)  # frames N, CA, C of each residue
    natoms = torch.from_numpy(_NATOMS).to(dev)[types]
    first = natoms.cumsum(1) - natoms
    table = [_SIDE[c] for c in LETTERS] + [[]]
    spots, slots = [], []

    def put(x, slot, where):
        spots.append(x)
        slots.append(torch.where(where, first + slot, max_atoms))

    def local(frame, origin, v):
        return (frame @ v[..., None]).squeeze(-1) + origin

    def tensor(rows):
        return torch.tensor(rows, dtype=dt, device=dev)

    some = types < 20
    put(p[:, :, 0], 0, some)
    put(p[:, :, 1], 1, some)
    put(p[:, :, 2], natoms - 2, some)
    put(local(R[:, :, 2], p[:, :, 2], tensor(_CO)), natoms - 1, some)
    for k, v in enumerate(_PRO):
        put(local(R[:, :, 1], p[:, :, 1], tensor(v)), 2 + k, types == LETTERS.index("P"))
    c, s = math.cos(_DUMMY), math.sin(_DUMMY)
    S, o = R[:, :, 1] @ tensor([[1, 0, 0], [0, c, -s], [0, s, c]]), p[:, :, 1]
    for k in range(5):
        joint = [t[k] if len(t) > k else (0.0, 0.0, []) for t in table]
        beta, d = tensor([j[0] for j in joint])[types], tensor([j[1] for j in joint])[types]
        turns = torch.tensor([len(t) > k and c != "A" for t, c in zip(table, LETTERS + "-")], device=dev)[types]
        cb, sb = torch.cos(beta), torch.sin(beta)
        o = o + d[..., None] * (S @ torch.stack([cb, torch.zeros_like(cb), -sb], -1)[..., None]).squeeze(-1)
        S = S @ _turn(ang[:, 3 + k] * turns, cb, sb)
        before = [2 + sum(len(j[2]) for j in t[:k]) for t in table]
        for a in range(max(len(j[2]) for j in joint)):
            v = tensor([j[2][a] if len(j[2]) > a else (0.0, 0.0, 0.0) for j in joint])[types]
            has = torch.tensor([len(j[2]) > a for j in joint], device=dev)[types]
            put(local(S, o, v), torch.tensor([n + a for n in before], device=dev)[types], has)
    spots, slots = torch.cat(spots, 1), torch.cat(slots, 1)
    out = torch.zeros(B, max_atoms + 1, 3, dtype=dt, device=dev)
    return out.scatter(1, slots[..., None].expand(-1, -1, 3), spots)[:, :-1].reshape(B, 3 * max_atoms)


def _rmsd(x, y, num_atoms):
    """Least RMSD of rows [B, 3N] after centring both, and the (transposed) rotation that gives it."""
    B, n = x.shape[0], num_atoms.to(x.dtype)
    keep = (torch.arange(x.shape[1] // 3, device=x.device)[None, :] < num_atoms[:, None])[..., None]
    x, y = x.view(B, -1, 3) * keep, y.view(B, -1, 3) * keep
    x = (x - x.sum(1, keepdim=True) / n[:, None, None]) * keep
    y = (y - y.sum(1, keepdim=True) / n[:, None, None]) * keep
    r = x.transpose(1, 2) @ y
    a, b, c, d, e, f, g, h, i = r.reshape(B, 9).unbind(1)
    key = torch.stack([a + e + i, f - h, g - c, b - d, f - h, a - e - i, b + d, c + g, g - c, b + d, e - a - i, f + h,
                       b - d, c + g, f + h, i - a - e], 1).view(B, 4, 4)
    lam, vec = torch.linalg.eigh(key)
    q0, q1, q2, q3 = vec[:, :, -1].detach().unbind(1)
    turn = torch.stack([q0 * q0 + q1 * q1 - q2 * q2 - q3 * q3, 2 * (q1 * q2 + q0 * q3), 2 * (q1 * q3 - q0 * q2),
                        2 * (q1 * q2 - q0 * q3), q0 * q0 - q1 * q1 + q2 * q2 - q3 * q3, 2 * (q2 * q3 + q0 * q1),
                        2 * (q1 * q3 + q0 * q2), 2 * (q2 * q3 - q0 * q1), q0 * q0 - q1 * q1 - q2 * q2 + q3 * q3], 1)
    return torch.sqrt(((x * x).sum((1, 2)) + (y * y).sum((1, 2)) - 2 * lam[:, -1] + 1e-10) / n), turn.view(B, 3, 3)


def exact(case, seed):
    kind, s = case["kind"], _inputs(case, seed)
    if kind == "typed":  # values copied to other places, nothing computed
        return None
    if kind in ("backbone", "fullatom", "train"):
        ang = s["angles"].double().requires_grad_(case["grad"])
        if kind == "backbone":
            out = _backbone(ang, s["lengths"])
        else:
            out = _full_atom(ang, s["types"], s["max_atoms"])
        first = [out.detach()] if kind == "backbone" else [out.detach(), None, None, None]
        if kind == "train":
            rmsd = _rmsd(out, s["target"].double(), s["num_atoms"])[0]
            return [rmsd.detach(), torch.autograd.grad(rmsd.mean(), ang)[0]]
        if not case["grad"]:
            return first
        return first + [torch.autograd.grad(out, ang, s["up"].double())[0]]
    if kind == "score":
        return list(_rmsd(s["coords"].double(), s["target"].double(), s["num_atoms"]))
    B = case["batch"]
    keep, rot = s["real"][..., None], s["rot"].double()
    x = s["coords"].double().view(B, -1, 3)
    center = x.sum(1) / s["num_atoms"][:, None]
    turned = ((x - center[:, None]) @ rot.transpose(1, 2)) * keep
    inf = torch.full_like(turned, math.inf)
    back = (s["up"].double().view(B, -1, 3) * keep) @ rot
    return [center, turned.reshape(B, -1), torch.where(keep, turned, inf).amin(1), torch.where(keep, turned, -inf).amax(1),
            back.reshape(B, -1)]
