"""CoordsTransform on the GPU against the oracle (restatement of
Layers/FullAtomModel/TransformCUDAKernels.cu:4-107 and Math/nUtil.cpp:27-57).

Tolerances: translate and its backward are single additions (bit-exact in both
dtypes); rotate 1e-12 (FP64) / 2e-6 (FP32) relative to the coordinate scale;
centre 1e-12 / 1e-6 (FP64 accumulation in the kernel); bounding box bit-exact."""
import ctypes

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def case(dtype, B=9, S=700, seed=0):
    rng = np.random.default_rng(seed)
    x = (rng.standard_normal((B, 3 * S)) * 30).astype(np.float64)
    na = rng.integers(0, S + 1, B).astype(np.int32)
    na[0], na[1], na[2] = S, 0, 1
    T = rng.standard_normal((B, 3)) * 10
    R = oracle.rotation_from_u(rng.uniform(0, 1, (B, 3)))
    if dtype == torch.float32:
        x, T, R = x.astype(np.float32), T.astype(np.float32), R.astype(np.float32)
    return x, na, T, R


@pytest.fixture(scope="module")
def ct(built):
    from torchproteinlibrary_gb300.FullAtomModel import CoordsTransform
    return CoordsTransform


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_translate_rotate_center_layers(ct, dtype):
    x, na, T, R = case(dtype)
    dev = torch.device("cuda")
    xt = torch.tensor(x, device=dev, requires_grad=True)
    nat = torch.tensor(na)
    tol_rot = 2e-6 if dtype == torch.float32 else 1e-12
    scale = np.abs(x).max()

    y = ct.CoordsTranslate()(xt, torch.tensor(T, device=dev), nat)
    assert np.array_equal(y.detach().cpu().numpy(), oracle.coords_translate(x, T, na))
    g = torch.tensor(np.random.default_rng(1).standard_normal(x.shape).astype(x.dtype), device=dev)
    y.backward(g)
    assert np.array_equal(xt.grad.cpu().numpy(), oracle.coords_translate(g.cpu().numpy(), None, na))

    xt.grad = None
    y = ct.CoordsRotate()(xt, torch.tensor(R, device=dev), nat)
    assert np.abs(y.detach().cpu().numpy() - oracle.coords_rotate(x, R, na)).max() <= tol_rot * scale
    y.backward(g)
    gref = oracle.coords_rotate(g.cpu().numpy(), R, na, transpose=True)
    assert np.abs(xt.grad.cpu().numpy() - gref).max() <= tol_rot * np.abs(gref).max()

    xt.grad = None
    c = ct.Coords2Center()(xt, nat)
    tol_c = 1e-6 if dtype == torch.float32 else 1e-12
    assert np.abs(c.detach().cpu().numpy() - oracle.coords_center(x, na)).max() <= tol_c * scale
    gc = torch.tensor(np.random.default_rng(2).standard_normal((x.shape[0], 3)).astype(x.dtype), device=dev)
    c.backward(gc)
    gref = oracle.coords_center_backward(gc.cpu().numpy(), na, x.shape[1] // 3)
    assert np.allclose(xt.grad.cpu().numpy(), gref, rtol=1e-6 if dtype == torch.float32 else 1e-14, atol=0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_bbox_and_centering_composition(ct, dtype):
    """getBBox against the oracle; translating by minus the centre centres the chain
    (the reference's Coords2Center + CoordsTranslate idiom)."""
    x, na, _, _ = case(dtype, seed=4)
    dev = torch.device("cuda")
    xt = torch.tensor(x, device=dev)
    lo, hi = ct.getBBox(xt, torch.tensor(na))
    rlo, rhi = oracle.coords_bbox(x, na)
    assert np.array_equal(lo.cpu().numpy(), rlo) and np.array_equal(hi.cpu().numpy(), rhi)
    c = ct.Coords2Center()(xt, torch.tensor(na))
    y = ct.CoordsTranslate()(xt, -c, torch.tensor(na))
    c2 = ct.Coords2Center()(y, torch.tensor(na)).cpu().numpy()
    assert np.abs(c2).max() <= (1e-4 if dtype == torch.float32 else 1e-11)


def test_c_abi_translate_rotate(built):
    from torchproteinlibrary_gb300 import capi
    lib = capi.lib()
    x, na, T, R = case(torch.float32, B=5, S=33, seed=7)
    dev = torch.device("cuda")
    xt = torch.tensor(x, device=dev)
    nat = torch.tensor(na, device=dev)
    out = torch.full_like(xt, float("nan"))
    capi.check(lib.tpl_coords_translate_f32(xt.data_ptr(), out.data_ptr(), torch.tensor(T, device=dev).data_ptr(),
                                            nat.data_ptr(), 5, 33, capi.stream_ptr()), "translate")
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), oracle.coords_translate(x, T, na))
    Rt = torch.tensor(R, device=dev)
    capi.check(lib.tpl_coords_rotate_f32(xt.data_ptr(), out.data_ptr(), Rt.data_ptr(), 0, nat.data_ptr(), 5, 33,
                                         capi.stream_ptr()), "rotate")
    torch.cuda.synchronize()
    assert np.abs(out.cpu().numpy() - oracle.coords_rotate(x, R, na)).max() <= 2e-6 * np.abs(x).max()
    assert lib.tpl_coords_rotate_f32(None, out.data_ptr(), Rt.data_ptr(), 0, nat.data_ptr(), 5, 33, None) == -1


@pytest.mark.parametrize("S", [700, 33, 4000])
def test_center_vector_and_scalar_paths(ct, S):
    """Coords2Center in float32 reads 16-byte rows (stride a multiple of 4 atoms) as
    float4 groups of four atoms plus a scalar tail, and other strides atom by atom;
    both against the oracle within 1e-6 of the coordinate scale, with counts of every
    residue mod 4 and a chain far from the origin."""
    x, na, _, _ = case(torch.float32, B=12, S=S, seed=11)
    na[3:7] = [max(0, S - 1), max(0, S - 2), max(0, S - 3), min(5, S)]
    x[4] += 500.0
    c = ct.Coords2Center()(torch.tensor(x, device="cuda"), torch.tensor(na)).cpu().numpy()
    assert np.abs(c - oracle.coords_center(x, na)).max() <= 1e-6 * np.abs(x).max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("S,offs", [(1, (0, 0)), (3, (0, 0)), (5, (1, 1)), (127, (0, 0)), (128, (2, 2)), (129, (3, 3)),
                                    (130, (0, 0)), (131, (0, 1)), (1027, (0, 0))])
def test_rows_at_every_alignment(ct, dtype, S, offs):
    """Rows that start at every place of a 16-byte block (odd strides, storage offsets of
    the input and, through the extension entries, of the output, alike or not) and sizes
    around the vector groups and warp tiles, with every count from 0 to 9 atoms and a full
    row: translate, its backward, the centre's backward and the box bit for bit; rotate and
    centre to the tolerances of the file."""
    from torchproteinlibrary_gb300 import load_extension
    fm = load_extension("_FullAtomModel")
    x, na, T, R = case(dtype, B=14, S=S, seed=S)
    na[:] = np.minimum(np.arange(14) - 1, S)
    na[0] = na[13] = S
    dev, scale = torch.device("cuda"), np.abs(x).max()

    def at(v, off):
        v = np.asarray(v)
        t = torch.empty(v.size + off, dtype=dtype, device=dev)[off:].view(v.shape)
        return t.copy_(torch.tensor(v))

    xt, nat, Tt, Rt = at(x, offs[0]), torch.tensor(na, device=dev), at(T, 0), at(R, 0)
    out = at(np.full_like(x, 7.0), offs[1])
    fm.CoordsTranslateGPU_forward(xt, out, Tt, nat)
    assert np.array_equal(out.cpu().numpy(), oracle.coords_translate(x, T, na))
    fm.CoordsTranslateGPU_backward(xt, out, Tt, nat)
    assert np.array_equal(out.cpu().numpy(), oracle.coords_translate(x, None, na))
    tol = 2e-6 if dtype == torch.float32 else 1e-12
    fm.CoordsRotateGPU_forward(xt, out, Rt, nat)
    assert np.abs(out.cpu().numpy() - oracle.coords_rotate(x, R, na)).max() <= tol * scale
    fm.CoordsRotateGPU_backward(xt, out, Rt, nat)
    assert np.abs(out.cpu().numpy() - oracle.coords_rotate(x, R, na, transpose=True)).max() <= tol * scale
    c = ct.Coords2Center()(xt, nat)
    assert np.abs(c.cpu().numpy() - oracle.coords_center(x, na)).max() <= (1e-6 if dtype == torch.float32 else 1e-12) * scale
    fm.Coords2CenterGPU_backward(Tt, out, nat)
    assert np.allclose(out.cpu().numpy(), oracle.coords_center_backward(T, na, S),
                       rtol=1e-6 if dtype == torch.float32 else 1e-14, atol=0)
    a, b = ct.getBBox(xt, nat)
    ra, rb = oracle.coords_bbox(x, na)
    assert np.array_equal(a.cpu().numpy(), ra) and np.array_equal(b.cpu().numpy(), rb)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("S,offs", [(299, (0, 0)), (301, (1, 1)), (1499, (0, 0)), (1500, (2, 2)), (1501, (0, 0)),
                                    (1502, (3, 3)), (1503, (0, 1)), (12001, (0, 0))])
def test_large_batches(ct, dtype, S, offs):
    """Batches large enough for what small ones do not take: shifts as vectors between the
    boundaries of rows that start anywhere, rotations in tiles (float32), reductions by 128
    threads; rows on both sides of each line and at every 16-byte phase, input and output in
    different phases, counts from none to 9 atoms and full rows.  Translate, the two shift
    backwards and the box bit for bit; rotate and centre to the tolerances of the file."""
    from torchproteinlibrary_gb300 import load_extension
    fm = load_extension("_FullAtomModel")
    K, B = 17, 3400 if S < 12000 else 700
    x, na, T, R = case(dtype, B=K, S=S, seed=S)
    na[:] = np.minimum(np.arange(K) - 1, S)
    na[0], na[11:] = S, [S, S - 1, S - 2, S - 3, S - 5, S // 2]
    dev, scale = torch.device("cuda"), np.abs(x).max()
    rows = torch.arange(B, device=dev) % K

    def at(v, off):
        v = torch.tensor(np.asarray(v), device=dev)
        t = torch.empty(B * v[0].numel() + off, dtype=dtype, device=dev)[off:].view(B, *v.shape[1:])
        return t.copy_(v[rows])

    def same(got, want):
        return torch.equal(got, torch.tensor(want, device=dev)[rows])

    def error(got, want):
        return (got - torch.tensor(want, device=dev)[rows]).abs().max().item()

    xt, nat, Tt, Rt = at(x, offs[0]), torch.tensor(na, device=dev)[rows].contiguous(), at(T, 0), at(R, 0)
    out = at(np.full_like(x, 7.0), offs[1])
    fm.CoordsTranslateGPU_forward(xt, out, Tt, nat)
    assert same(out, oracle.coords_translate(x, T, na))
    fm.CoordsTranslateGPU_backward(xt, out, Tt, nat)
    assert same(out, oracle.coords_translate(x, None, na))
    tol = 2e-6 if dtype == torch.float32 else 1e-12
    for call, transpose in ((fm.CoordsRotateGPU_forward, False), (fm.CoordsRotateGPU_backward, True)):
        out.fill_(7.0)
        call(xt, out, Rt, nat)
        assert error(out, oracle.coords_rotate(x, R, na, transpose=transpose)) <= tol * scale
        assert not out[1].any()
    c = ct.Coords2Center()(xt, nat)
    assert error(c, oracle.coords_center(x, na)) <= (1e-6 if dtype == torch.float32 else 1e-12) * scale
    fm.Coords2CenterGPU_backward(Tt, out, nat)
    want = torch.tensor(oracle.coords_center_backward(T, na, S), device=dev)[rows]
    assert torch.allclose(out, want, rtol=1e-6 if dtype == torch.float32 else 1e-14, atol=0)
    lo, hi = ct.getBBox(xt, nat)
    rlo, rhi = oracle.coords_bbox(x, na)
    assert same(lo, rlo) and same(hi, rhi)
