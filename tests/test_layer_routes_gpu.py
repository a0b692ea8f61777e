"""The CoordsTransform and Coords2TypedCoords modules run the extension's C++ autograd
functions; the Python functions of the same name stay, and take the calls that are traced.
Both routes give the same outputs and gradients bit for bit, for counts on the device or on
the host, and for inputs that are not contiguous."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fa(built):
    names = ("FullAtomModel", "FullAtomModel.CoordsTransform.CoordsTransform",
             "FullAtomModel.Coords2TypedCoords.Coords2TypedCoords")
    return [importlib.import_module("torchproteinlibrary_gb300." + n) for n in names]


def _inputs(dtype, strided):
    g = torch.Generator("cuda").manual_seed(3)
    B, S = 5, 41
    x = torch.randn(B, 3 * S, dtype=dtype, device="cuda", generator=g) * 20
    if strided:
        x = torch.cat([x, x], 1)[:, ::2]  # another tensor, its rows strided
    na = torch.tensor([41, 0, 1, 17, 40], dtype=torch.int32)
    return x, na, torch.randn(x.shape, dtype=dtype, device="cuda", generator=g), g


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("host_counts", [False, True])
def test_transform_modules_match_functions(fa, dtype, strided, host_counts):
    _, ct, _ = fa
    x, na, up, g = _inputs(dtype, strided)
    if not host_counts:
        na = na.cuda()
    T = torch.randn(5, 3, dtype=torch.float64, device="cuda", generator=g)
    R = ct.getRotation(torch.rand(5, 3, dtype=torch.float64, device="cuda", generator=g))
    for module, function, args in ((ct.CoordsTranslate(), ct.CoordsTranslateFunction, (T, na)),
                                   (ct.CoordsRotate(), ct.CoordsRotateFunction, (R, na)),
                                   (ct.Coords2Center(), ct.Coords2CenterFunction, (na,))):
        got, want = [], []
        for call, out in ((module, got), (function.apply, want)):
            leaf = x.clone().requires_grad_() if not strided else x.detach().requires_grad_()
            y = call(leaf, *args)
            u = up if y.shape == up.shape else up[:, :3].contiguous()
            out += [y.detach(), torch.autograd.grad(y, leaf, u)[0]]
        assert "CppNode" in module(x.clone().requires_grad_(), *args).grad_fn.name()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    lo, hi = ct.getBBox(x, na)
    keep = torch.arange(41, device="cuda")[None, :] < na.cuda()[:, None]
    v = x.reshape(5, 41, 3)
    assert torch.equal(lo, torch.where(keep[..., None], v, torch.full_like(v, float("inf"))).amin(1))
    assert torch.equal(hi, torch.where(keep[..., None], v, torch.full_like(v, float("-inf"))).amax(1))


def test_modules_refuse_what_the_functions_refuse(fa):
    _, ct, _ = fa
    x, na, _, _ = _inputs(torch.float32, False)
    with pytest.raises(ValueError):
        ct.CoordsTranslate()(x.view(5, 41, 3), x[:, :3], na)
    with pytest.raises(RuntimeError):
        ct.CoordsRotate()(x.cpu(), torch.eye(3).repeat(5, 1, 1), na)
    with pytest.raises(RuntimeError):
        ct.Coords2Center()(x[:, :-1], na)


def test_tracing_takes_the_python_functions(fa):
    _, ct, _ = fa
    x, na, _, _ = _inputs(torch.float32, False)
    T, nad = torch.randn(5, 3, device="cuda"), na.cuda()
    seen = []
    original = ct.CoordsTranslateFunction.apply
    ct.CoordsTranslateFunction.apply = staticmethod(lambda *a: seen.append(1) or original(*a))
    try:
        torch.jit.trace(lambda v: ct.CoordsTranslate()(v, T, nad), x, check_trace=False)
    finally:
        ct.CoordsTranslateFunction.apply = original
    assert seen


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_typed_module_matches_function(fa, dtype):
    fam, _, tc = fa
    rng = np.random.default_rng(9)
    seqs = ["".join(rng.choice(list("ACDEFGHIKLMNPQRSTVWY"), n)) for n in (30, 1, 77)]
    ang = torch.randn(3, 8, 77, dtype=dtype, device="cuda")
    coords, rn, an, na = fam.Angles2Coords()(ang, seqs)
    results = []
    for call in (fam.Coords2TypedCoords(), tc.Coords2TypedCoordsFunction.apply):
        for counts in (na, na.cuda()):
            x = coords.detach().clone().requires_grad_()
            out, n, off = call(x, rn, an, counts)
            grad, = torch.autograd.grad(out, x, torch.cos(out.detach()))
            results.append((out.detach(), n, off, grad))
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))


@pytest.mark.parametrize("B,L,fills", [(2048, 517, 0), (64, 999, 0), (1024, 700, 0), (3, 5001, 1)])
def test_captured_backbone_step_fills_only_what_is_read(built, monkeypatch, B, L, fills):
    """A captured Angles2Backbone step zeroes its workspace only where chains are split into
    tiles (few chains of more than 4096 residues), whatever names the scheme: the tuned
    table, or the library's rule for rows of odd length and shapes outside the table.  Three
    replays equal the eager step (bit for bit where chains stay whole)."""
    m = importlib.import_module("torchproteinlibrary_gb300.ReducedModel.Angles2Backbone.Angles2Backbone")
    g = torch.Generator("cuda").manual_seed(L)
    ang = ((torch.rand(B, 3, L, device="cuda", generator=g) * 2 - 1) * np.pi).requires_grad_()
    lengths = torch.randint(1, L + 1, (B,), device="cuda", generator=g, dtype=torch.int32)
    up = torch.randn(B, 9 * L, device="cuda", generator=g)
    layer = m.Angles2Backbone()

    def step():
        coords = layer(ang, lengths)
        return coords, torch.autograd.grad(coords, ang, up)[0]

    want = [t.detach().clone() for t in step()]
    calls, original = [], m.new_workspace
    monkeypatch.setattr(m, "new_workspace", lambda *a: calls.append(a) or original(*a))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    calls.clear()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    assert len(calls) == fills
    for _ in range(3):
        for t in out:
            t.detach().fill_(float("nan"))
        graph.replay()
        for t, w in zip(out, want):
            if fills:  # the look-back's order, and with it the rounding, may differ
                assert (t.detach() - w).abs().max() <= 1e-4 * w.abs().max()
            else:
                assert torch.equal(t.detach(), w)


def test_backbone_names_functorch_in_its_refusal(built):
    """float32 Angles2Backbone does not run under functorch transforms, and says so."""
    from torchproteinlibrary_gb300.ReducedModel import Angles2Backbone
    layer, n = Angles2Backbone(), torch.tensor([8, 5], dtype=torch.int32, device="cuda")
    angles = torch.randn(2, 3, 8, device="cuda")
    with pytest.raises(RuntimeError, match="functorch"):
        torch.func.grad(lambda a: layer(a, n).sum())(angles)
    with pytest.raises(RuntimeError, match="functorch"):
        torch.func.vmap(lambda a: layer(a, n))(torch.stack([angles, angles]))
