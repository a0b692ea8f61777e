"""Coords2RMSD on the GPU (the loss of the training-step workload).

The reference's _RMSD extension does not build against torch 2.x (Tensor::eig was
removed), so the oracle is a numpy restatement of its CPU path; it is pinned by the
properties the reference's own tests check (UnitTests/RMSD/Coords2RMSD/test.py:
RMSD of a rigidly moved copy is 0, gradcheck).  Tolerances: FP64 1e-9 relative,
FP32 1e-4 relative (rmsd) and 1e-3 relative (gradients)."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def random_rotation(rng):
    q = rng.standard_normal(4)
    q /= np.linalg.norm(q)
    a, b, c, d = q
    return np.array([[a * a + b * b - c * c - d * d, 2 * (b * c - a * d), 2 * (b * d + a * c)],
                     [2 * (b * c + a * d), a * a - b * b + c * c - d * d, 2 * (c * d - a * b)],
                     [2 * (b * d - a * c), 2 * (c * d + a * b), a * a - b * b - c * c + d * d]])


def case(B=8, N=300, seed=0):
    rng = np.random.default_rng(seed)
    na = rng.integers(3, N + 1, B).astype(np.int32)
    src = rng.standard_normal((B, 3 * N)) * 10
    dst = rng.standard_normal((B, 3 * N)) * 10
    return src, dst, na


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-9), (torch.float32, 1e-4)])
def test_matches_oracle(built, dtype, tol):
    from torchproteinlibrary_gb300.RMSD import Coords2RMSD
    src, dst, na = case()
    layer = Coords2RMSD()
    x = torch.tensor(src, dtype=dtype, device="cuda", requires_grad=True)
    y = torch.tensor(dst, dtype=dtype, device="cuda")
    r = layer(x, y, torch.tensor(na, device="cuda"))
    r.sum().backward()
    ro, UTo, go = oracle.rmsd(src, dst, na)
    assert np.allclose(r.detach().double().cpu().numpy(), ro, rtol=tol, atol=0)
    g = x.grad.double().cpu().numpy()
    assert np.abs(g - go).max() <= 10 * tol * np.abs(go).max()
    # UT agrees up to the sign convention of the eigenvector (U(q) = U(-q))
    assert np.allclose(layer.UT.double().cpu().numpy(), UTo, atol=100 * tol)


def test_rigid_copy_has_zero_rmsd(built):
    """UnitTests/RMSD/Coords2RMSD/test.py: a rotated and translated copy gives RMSD ~ 0."""
    from torchproteinlibrary_gb300.RMSD import Coords2RMSD
    rng = np.random.default_rng(1)
    B, N = 6, 200
    src = rng.standard_normal((B, N, 3)) * 15
    dst = np.stack([src[b] @ random_rotation(rng).T + rng.standard_normal(3) * 20 for b in range(B)])
    na = np.full(B, N, np.int32)
    r = Coords2RMSD()(torch.tensor(src.reshape(B, -1), device="cuda"), torch.tensor(dst.reshape(B, -1), device="cuda"),
                      torch.tensor(na, device="cuda"))
    assert r.max().item() < 1e-4


def test_gradcheck_and_function_api(built):
    from torchproteinlibrary_gb300.RMSD import Coords2RMSD
    from torchproteinlibrary_gb300.RMSD.Coords2RMSD import Coords2RMSDFunction
    src, dst, na = case(B=3, N=12, seed=5)
    x = torch.tensor(src, device="cuda", requires_grad=True)
    y = torch.tensor(dst, device="cuda")
    n = torch.tensor(na, device="cuda")
    assert torch.autograd.gradcheck(lambda a: Coords2RMSD()(a, y, n), (x,), eps=1e-6, atol=1e-6, rtol=1e-5)
    # Function API on already-centred inputs (reference Coords2RMSDFunction)
    xc = x.detach().clone()
    yc = y.clone()
    for b in range(3):
        m = na[b]
        xc[b, :3 * m] -= xc[b, :3 * m].view(m, 3).mean(0).repeat(m)
        yc[b, :3 * m] -= yc[b, :3 * m].view(m, 3).mean(0).repeat(m)
    r1, UT = Coords2RMSDFunction.apply(xc, yc, n)
    r2 = Coords2RMSD()(x.detach(), y, n)
    assert torch.allclose(r1, r2, rtol=1e-9)


def test_host_num_atoms_reused_and_refreshed(built):
    """A host num_atoms tensor is copied to the device once and reused on later calls;
    changing it in place makes the next call copy the new counts."""
    from torchproteinlibrary_gb300.RMSD import Coords2RMSD
    src, dst, na = case(B=4, N=50, seed=3)
    layer = Coords2RMSD()
    x = torch.tensor(src, device="cuda")
    y = torch.tensor(dst, device="cuda")
    n = torch.tensor(na, dtype=torch.int32)
    r1 = layer(x, y, n)
    r2 = layer(x, y, n)
    assert torch.equal(r1, r2)
    n[0] = 3
    r3 = layer(x, y, n)
    ref, _, _ = oracle.rmsd(src, dst, n.numpy())
    assert np.allclose(r3.cpu().numpy(), ref, rtol=1e-9, atol=0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_small_and_degenerate_chains(built, dtype):
    """Chains of 0, 1, 2 and 3 atoms, collinear and planar chains (repeated
    eigenvalues of the key matrix), identical structures (rmsd 0) and a mirrored copy:
    rmsd against the oracle, finite gradients everywhere and zero gradient past each
    chain.  rmsd = sqrt((R2 - 2 lambda + 1e-10) / N) cancels for near-identical
    structures, so its absolute resolution is about sqrt(eps R2 / N): the tolerance is
    2e-2 A in float32 and 1e-5 A in float64 (coordinates of about 10 A here)."""
    from torchproteinlibrary_gb300.RMSD import Coords2RMSD
    rng = np.random.default_rng(77)
    N = 40
    src = rng.standard_normal((10, N, 3)) * 8
    dst = rng.standard_normal((10, N, 3)) * 8
    na = np.array([0, 1, 2, 3, N, N, N, N, N, N], np.int32)
    line = np.linspace(-20, 20, N)[:, None] * np.array([0.3, 0.5, 0.8])
    src[4], dst[4] = line, line[::-1] + 5.0                      # collinear
    src[5, :, 2] = 0.0
    dst[5] = src[5] @ random_rotation(rng).T + 3.0                # planar, rigid copy
    dst[6] = src[6]                                               # identical
    dst[7] = src[7] * np.array([-1.0, 1.0, 1.0])                  # mirror image
    src[8, :, 2] = 0.0
    dst[8, :, 2] = 0.0                                            # both planar
    x = torch.tensor(src.reshape(10, -1), dtype=dtype, device="cuda", requires_grad=True)
    y = torch.tensor(dst.reshape(10, -1), dtype=dtype, device="cuda")
    r = Coords2RMSD()(x, y, torch.tensor(na, device="cuda"))
    r.sum().backward()
    ro, _, _ = oracle.rmsd(src.reshape(10, -1), dst.reshape(10, -1), na)
    atol = 2e-2 if dtype == torch.float32 else 1e-5
    np.testing.assert_allclose(r.detach().double().cpu().numpy(), ro, atol=atol, rtol=0)
    g = x.grad.double().cpu().numpy()
    assert np.isfinite(g).all()
    for b in range(10):
        assert np.all(g[b, 3 * na[b]:] == 0.0)


def _at_offset(v, off, dtype):
    """A contiguous CUDA tensor of v whose storage starts `off` elements into an allocation."""
    t = torch.empty(v.size + off, dtype=dtype, device="cuda")[off:].view(v.shape)
    t.copy_(torch.tensor(v, dtype=dtype))
    return t


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("B,N,offs", [(40, 41, (0, 0)), (40, 42, (1, 1)), (40, 43, (3, 3)), (40, 41, (0, 1)),
                                      (320, 61, (0, 0)), (620, 70, (2, 2)), (4, 4099, (0, 0))])
def test_atom_groups_at_every_alignment_and_block_size(built, dtype, B, N, offs):
    """Rows that start at every place of a 16-byte block (odd strides, offset storage, the
    two sets alike or not), counts from 1 atom up around the groups of four, and batches on
    both sides of each block size of the forward; rmsd, rotation-invariant gradient."""
    from torchproteinlibrary_gb300.RMSD import Coords2RMSD
    rng = np.random.default_rng(B + N)
    na = np.where(np.arange(B) < 24, np.arange(B) + 1, rng.integers(25, N + 1, B)).astype(np.int32)
    na[-1] = N
    src = rng.standard_normal((B, 3 * N)) * 10 + 30
    dst = rng.standard_normal((B, 3 * N)) * 10 - 20
    x = _at_offset(src, offs[0], dtype).requires_grad_()
    y = _at_offset(dst, offs[1], dtype)
    w = torch.rand(B, dtype=dtype, device="cuda", generator=torch.Generator("cuda").manual_seed(1)) + 0.5
    r = Coords2RMSD()(x, y, torch.tensor(na))
    g, = torch.autograd.grad(r, x, w)
    xs, ys = x.detach().double().cpu().numpy(), y.double().cpu().numpy()
    ref, _, grads = oracle.rmsd(xs, ys, na)
    # one or two atoms superpose exactly: there rmsd is 0 up to the rounding of the sums
    tol = 1e-4 if dtype == torch.float32 else 1e-9
    assert np.abs(r.detach().double().cpu().numpy() - ref)[na > 2].max() <= tol * ref.max()
    g = g.double().cpu().numpy()
    for b in range(B):
        assert not g[b, 3 * na[b]:].any()
        if na[b] < 8:  # nearly planar sets: the rotation is ill-conditioned
            continue
        n = int(na[b])
        want = float(w[b]) * grads[b, :3 * n]
        scale = np.abs(want).max()
        assert np.abs(g[b, :3 * n] - want).max() <= (1e-3 if dtype == torch.float32 else 1e-8) * scale


@pytest.mark.parametrize("half", [0, 1])
def test_two_chains_per_cta(built, half):
    """Large batches solve two chains per warp, one on each half: an odd batch (the last CTA
    has one chain), and next to an ordinary chain one that takes the degenerate solve (a
    rigid copy of a collinear set), an empty one and a one-atom one, on either half.
    Tolerance as for the other batches: 1e-4 of the largest value in float32."""
    from torchproteinlibrary_gb300.RMSD import Coords2RMSD
    rng = np.random.default_rng(7 + half)
    B, N = 4 * torch.cuda.get_device_properties(0).multi_processor_count + 5, 37
    B += 1 - B % 2
    na = rng.integers(9, N + 1, B).astype(np.int32)
    src = rng.standard_normal((B, 3 * N)) * 10 + 30
    dst = rng.standard_normal((B, 3 * N)) * 10 - 20
    for b in range(half, B - 1, 14):
        line = np.outer(np.arange(N), [1.0, 2.0, -0.5])
        src[b], dst[b] = line.ravel(), line[::-1].ravel()
    na[half + 2:B - 1:14] = 0
    na[half + 4:B - 1:14] = 1
    r = Coords2RMSD()(torch.tensor(src, dtype=torch.float32).cuda(), torch.tensor(dst, dtype=torch.float32).cuda(),
                      torch.tensor(na))
    src, dst = src.astype(np.float32).astype(np.float64), dst.astype(np.float32).astype(np.float64)
    ref, _, _ = oracle.rmsd(src, dst, na)
    ok = na > 1
    assert np.abs(r.double().cpu().numpy() - ref)[ok].max() <= 1e-4 * ref[ok].max()
    assert r[torch.tensor(na == 0)].eq(0).all()


@pytest.mark.parametrize("B", [20, 400, 700])
def test_sampled_atoms_that_are_outliers(built, B):
    """The float32 forward takes its sums from a centre found on 16 atoms spread over the
    chain: coils of 2300 atoms that have those 16 moved 300 A away, as the only ones, in every
    block size of the forward, next to ordinary chains.  The float32 tolerances of this file
    (rmsd 1e-4 relative, gradients 1e-3 of the largest)."""
    from torchproteinlibrary_gb300.RMSD import Coords2RMSD
    rng = np.random.default_rng(23)
    K, N = 20, 2300
    pick = [N * (2 * i + 1) // 32 for i in range(16)]
    src = np.cumsum(rng.standard_normal((K, N, 3)), 1) * 0.7
    src -= src.mean(1, keepdims=True)
    src[::2, pick] += rng.permuted(np.tile([300.0, 0.0, 0.0], (K // 2, 1, 1)), axis=2)
    dst = np.stack([s @ random_rotation(rng).T for s in src]) + rng.standard_normal(src.shape) * 1.2
    src, dst = (v.reshape(K, -1).astype(np.float32) for v in (src, dst))
    na = np.full(K, N, np.int32)
    ref, _, gref = oracle.rmsd(src.astype(np.float64), dst.astype(np.float64), na)
    x = torch.tensor(src, device="cuda").repeat(B // K, 1).requires_grad_()
    y = torch.tensor(dst, device="cuda").repeat(B // K, 1)
    r = Coords2RMSD()(x, y, torch.tensor(na).repeat(B // K))
    g, = torch.autograd.grad(r.sum(), x)
    err = np.abs(r.detach().double().cpu().numpy().reshape(-1, K) / ref - 1.0).max()
    assert err <= 1e-4, err
    ge = np.abs(g.double().cpu().numpy().reshape(-1, K, 3 * N) - gref).max() / np.abs(gref).max()
    assert ge <= 1e-3, ge
