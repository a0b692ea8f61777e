"""Coords2TypedCoords on the GPU against the oracle (restatement of
coords2typedcoords_interface.cpp and ProtUtil::get11AtomType).  Integer and byte
work plus coordinate copies: everything is compared bit-exactly."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

AA = "ACDEFGHIKLMNPQRSTVWY"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_forward_backward_match_oracle(built, dtype):
    from torchproteinlibrary_gb300.FullAtomModel import Angles2Coords, Coords2TypedCoords
    rng = np.random.default_rng(11)
    lengths = [60, 1, 37, 120, 5]
    seqs = ["".join(rng.choice(list(AA), n)) for n in lengths]
    seqs[0] = (AA * 3)[:60]
    L = max(lengths)
    ang = torch.tensor(rng.uniform(-np.pi, np.pi, (len(seqs), 8, L)), dtype=dtype, device="cuda")
    coords, rn, an, na = Angles2Coords()(ang, seqs)
    x = coords.detach().clone().requires_grad_()
    typed, counts, offsets = Coords2TypedCoords()(x, rn, an, na)
    xc, rc, ac = coords.detach().cpu().numpy(), rn.cpu().numpy(), an.cpu().numpy()
    rt, rcnt, roff, ridx = oracle.typed_coords(xc, rc, ac, na.numpy())
    assert np.array_equal(typed.detach().cpu().numpy(), rt)
    assert np.array_equal(counts.cpu().numpy(), rcnt) and np.array_equal(offsets.cpu().numpy(), roff)
    g = torch.tensor(rng.standard_normal(typed.shape), dtype=dtype, device="cuda")
    typed.backward(g)
    ref = oracle.typed_coords_backward(g.cpu().numpy(), rcnt, ridx, xc.shape[1] // 3)
    assert np.array_equal(x.grad.cpu().numpy(), ref)


def test_unknown_name_is_reported(built):
    from torchproteinlibrary_gb300 import capi
    lib = capi.lib()
    dev = torch.device("cuda")
    x = torch.zeros(1, 6, device=dev)
    rn = torch.tensor([[list(b"ALA\0"), list(b"ALA\0")]], dtype=torch.uint8, device=dev)
    an = torch.tensor([[list(b"CB\0\0"), list(b"QQ\0\0")]], dtype=torch.uint8, device=dev)
    na = torch.tensor([2], dtype=torch.int32, device=dev)
    out = torch.empty(1, 6, device=dev)
    cnt = torch.empty(1, 11, dtype=torch.int32, device=dev)
    off = torch.empty_like(cnt)
    idx = torch.empty(1, 2, dtype=torch.int32, device=dev)
    ws = torch.zeros(64, dtype=torch.uint8, device=dev)
    capi.check(lib.tpl_typed_coords_forward_f32(x.data_ptr(), rn.data_ptr(), an.data_ptr(), na.data_ptr(), 1, 2, 2,
                                                out.data_ptr(), cnt.data_ptr(), off.data_ptr(), idx.data_ptr(),
                                                ws.data_ptr(), 64, capi.stream_ptr()), "typed")
    st = capi.ctypes.c_int()
    capi.check(lib.tpl_workspace_status(ws.data_ptr(), capi.stream_ptr(), capi.ctypes.byref(st)), "status")
    assert st.value == -10
    assert int(cnt.sum()) == 1 and int(cnt[0, 10]) == 1


def test_padded_names_take_the_slow_path(built):
    """Atom names with spaces or a tab inside their 4 bytes (PDB-style ' CA ', 'CB  ')
    are squeezed as the reference does (whitespace erased) and typed like the packed
    names; the packed names take the word-at-a-time path, the padded ones the byte
    loop.  Against the oracle, bit for bit."""
    from torchproteinlibrary_gb300 import capi
    lib = capi.lib()
    dev = torch.device("cuda")
    names = [b"N\0\0\0", b" CA ", b"C\0\0\0", b"O  \0", b"CB  ", b"\tCG\0", b"CD1\0", b"C D2", b"CE\0\0", b"NZ\0\0"]
    res = [b"LEU\0"] * 4 + [b"LEU\0", b"LEU\0", b"LEU\0", b"LEU\0", b"LYS\0", b"LYS\0"]
    n = len(names)
    rng = np.random.default_rng(5)
    x = torch.tensor(rng.standard_normal((1, 3 * n)), dtype=torch.float32, device=dev)
    rn = torch.tensor([[list(r) for r in res]], dtype=torch.uint8, device=dev)
    an = torch.tensor([[list(a) for a in names]], dtype=torch.uint8, device=dev)
    na = torch.tensor([n], dtype=torch.int32, device=dev)
    out = torch.full((1, 3 * n), float("nan"), device=dev)
    cnt = torch.empty(1, 11, dtype=torch.int32, device=dev)
    off = torch.empty_like(cnt)
    idx = torch.empty(1, n, dtype=torch.int32, device=dev)
    ws = torch.zeros(64, dtype=torch.uint8, device=dev)
    capi.check(lib.tpl_typed_coords_forward_f32(x.data_ptr(), rn.data_ptr(), an.data_ptr(), na.data_ptr(), 1, n, n,
                                                out.data_ptr(), cnt.data_ptr(), off.data_ptr(), idx.data_ptr(),
                                                ws.data_ptr(), 64, capi.stream_ptr()), "typed")
    st = capi.ctypes.c_int()
    capi.check(lib.tpl_workspace_status(ws.data_ptr(), capi.stream_ptr(), capi.ctypes.byref(st)), "status")
    assert st.value == 0
    rt, rcnt, roff, ridx = oracle.typed_coords(x.cpu().numpy(), rn.cpu().numpy(), an.cpu().numpy(), [n])
    assert int(rcnt.sum()) == n
    np.testing.assert_array_equal(cnt.cpu().numpy(), rcnt)
    np.testing.assert_array_equal(off.cpu().numpy(), roff)
    np.testing.assert_array_equal(idx.cpu().numpy(), ridx)
    np.testing.assert_array_equal(out.cpu().numpy(), rt)


def test_long_chain_path(built):
    """Rows of more than 32768 atoms take the one-CTA-per-chain kernel (no per-row type
    cache in shared memory): a 4100-residue chain beside a short one, forward and
    backward against the oracle bit for bit."""
    from torchproteinlibrary_gb300.FullAtomModel import Angles2Coords, Coords2TypedCoords
    rng = np.random.default_rng(17)
    seqs = ["".join(rng.choice(list(AA), 4100)), "".join(rng.choice(list(AA), 12))]
    ang = torch.tensor(rng.uniform(-np.pi, np.pi, (2, 8, 4100)), dtype=torch.float32, device="cuda")
    coords, rn, an, na = Angles2Coords()(ang, seqs)
    assert coords.shape[1] // 3 > 32768
    x = coords.detach().clone().requires_grad_()
    typed, counts, offsets = Coords2TypedCoords()(x, rn, an, na)
    xc, rc, ac = coords.detach().cpu().numpy(), rn.cpu().numpy(), an.cpu().numpy()
    rt, rcnt, roff, ridx = oracle.typed_coords(xc, rc, ac, na.numpy())
    assert np.array_equal(typed.detach().cpu().numpy(), rt)
    assert np.array_equal(counts.cpu().numpy(), rcnt) and np.array_equal(offsets.cpu().numpy(), roff)
    g = torch.tensor(rng.standard_normal(typed.shape), dtype=torch.float32, device="cuda")
    typed.backward(g)
    ref = oracle.typed_coords_backward(g.cpu().numpy(), rcnt, ridx, xc.shape[1] // 3)
    assert np.array_equal(x.grad.cpu().numpy(), ref)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("pad,na", [(p, [0, 1, 31, 32, 33, 127, 128, 129, 511, 512, 513, 640, 1025]) for p in range(4)] +
                         [(0, [16384, 3]), (1, [16384, 200]), (0, [20000])])
def test_groups_and_row_phases(built, dtype, pad, na):
    """Chains around the 128-atom groups and the split over four warps (eight past 16384
    atoms of row), rows at every 16-byte phase (odd strides), typed rows narrower than the
    input rows: counts, offsets, indexes and coordinates against the oracle, bit for bit."""
    from torchproteinlibrary_gb300 import load_extension
    fm = load_extension("_FullAtomModel")
    rng = np.random.default_rng(40 + pad)
    pairs = [(b"ALA\0", a) for a in (b"N\0\0\0", b"CA\0\0", b"CB\0\0", b"C\0\0\0", b"O\0\0\0")]
    pairs += [(b"LYS\0", b"NZ\0\0"), (b"CYS\0", b"SG\0\0"), (b"TRP\0", b"NE1\0"), (b"SER\0", b"OG\0\0"),
              (b"ASP\0", b"OD1\0"), (b"PHE\0", b"CZ\0\0"), (b"ARG\0", b"NH1\0")]
    na = np.array(na, np.int32)
    B, S_out = len(na), int(na.max())
    S = S_out + pad
    pick = rng.integers(0, len(pairs), (B, S))
    rn = np.array([[list(pairs[k][0]) for k in row] for row in pick], np.uint8)
    an = np.array([[list(pairs[k][1]) for k in row] for row in pick], np.uint8)
    x = rng.standard_normal((B, 3 * S)).astype(np.float32 if dtype == torch.float32 else np.float64)
    dev = torch.device("cuda")
    xt, rt, at = torch.tensor(x, device=dev), torch.tensor(rn, device=dev), torch.tensor(an, device=dev)
    out = torch.full((B, 3 * S_out), float("nan"), dtype=dtype, device=dev)
    cnt = torch.empty(B, 11, dtype=torch.int32, device=dev)
    off, idx = torch.empty_like(cnt), torch.full((B, S_out), -7, dtype=torch.int32, device=dev)
    fm.Coords2TypedCoords_forward(xt, rt, at, torch.tensor(na, device=dev), out, cnt, off, idx)
    want, wcnt, woff, widx = oracle.typed_coords(x, rn, an, na)
    assert np.array_equal(cnt.cpu().numpy(), wcnt) and np.array_equal(off.cpu().numpy(), woff)
    assert np.array_equal(out.cpu().numpy(), want) and np.array_equal(idx.cpu().numpy(), widx)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("pad", range(4))
def test_four_warps_in_large_batches(built, dtype, pad):
    """Batches of four chains per SM and more take four warps per chain: the same chains over
    and over, lengths around the tiles and groups, rows at every 16-byte phase, bit for bit."""
    from torchproteinlibrary_gb300 import load_extension
    fm = load_extension("_FullAtomModel")
    rng = np.random.default_rng(60 + pad)
    pairs = [(b"GLY\0", a) for a in (b"N\0\0\0", b"CA\0\0", b"C\0\0\0", b"O\0\0\0")]
    pairs += [(b"LYS\0", b"NZ\0\0"), (b"MET\0", b"SD\0\0"), (b"HIS\0", b"CG\0\0"), (b"THR\0", b"OG1\0")]
    na = np.array([0, 1, 31, 33, 127, 128, 129, 511, 512, 513, 641], np.int32)
    S_out = int(na.max())
    S = S_out + pad
    pick = rng.integers(0, len(pairs), (len(na), S))
    rn = np.array([[list(pairs[k][0]) for k in row] for row in pick], np.uint8)
    an = np.array([[list(pairs[k][1]) for k in row] for row in pick], np.uint8)
    x = rng.standard_normal((len(na), 3 * S)).astype(np.float32 if dtype == torch.float32 else np.float64)
    want, wcnt, woff, widx = oracle.typed_coords(x, rn, an, na)
    reps = 4 * torch.cuda.get_device_properties(0).multi_processor_count // len(na) + 1
    dev = torch.device("cuda")

    def rows(v):
        t = torch.tensor(v, device=dev)
        return t.repeat(reps, *[1] * (t.dim() - 1))

    B = reps * len(na)
    out = torch.full((B, 3 * S_out), float("nan"), dtype=dtype, device=dev)
    cnt = torch.empty(B, 11, dtype=torch.int32, device=dev)
    off, idx = torch.empty_like(cnt), torch.full((B, S_out), -7, dtype=torch.int32, device=dev)
    fm.Coords2TypedCoords_forward(rows(x), rows(rn), rows(an), rows(na), out, cnt, off, idx)
    for got, ref in ((out, want), (cnt, wcnt), (off, woff), (idx, widx)):
        assert torch.equal(got, rows(ref).to(got.dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("S", [1, 31, 33, 128, 599, 600, 601])
def test_short_rows_in_large_batches(built, dtype, S):
    """Batches of three chains per SM and more take the scattering kernel on rows of up to 600
    atoms: one chain fewer and that many, rows on both sides of the line, counts from none
    to all of the row, typed rows narrower than the input rows, a name pair without a type
    (left out and reported); bit for bit against the oracle."""
    from torchproteinlibrary_gb300 import load_extension
    fm = load_extension("_FullAtomModel")
    rng = np.random.default_rng(S)
    pairs = [(b"GLY\0", a) for a in (b"N\0\0\0", b"CA\0\0", b"C\0\0\0", b"O\0\0\0")]
    pairs += [(b"LYS\0", b"NZ\0\0"), (b"MET\0", b"SD\0\0"), (b"HIS\0", b"CG\0\0"), (b"THR\0", b"OG1\0")]
    K, S_out = 19, max(1, S - 1)
    na = rng.integers(0, S_out + 1, K).astype(np.int32)
    na[:3] = 0, S_out, min(1, S_out)
    pick = rng.integers(0, len(pairs), (K, S))
    rn = np.array([[list(pairs[k][0]) for k in row] for row in pick], np.uint8)
    an = np.array([[list(pairs[k][1]) for k in row] for row in pick], np.uint8)
    x = rng.standard_normal((K, 3 * S)).astype(np.float32 if dtype == torch.float32 else np.float64)
    want, wcnt, woff, widx = oracle.typed_coords(x, rn, an, na)
    wide = want.shape[1] // 3
    dev = torch.device("cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for B in (3 * sms - 1, 3 * sms):
        at = torch.arange(B, device=dev) % K

        def rows(v):
            return torch.tensor(v, device=dev)[at].contiguous()

        out = torch.full((B, 3 * S_out), float("nan"), dtype=dtype, device=dev)
        cnt = torch.empty(B, 11, dtype=torch.int32, device=dev)
        off, idx = torch.empty_like(cnt), torch.full((B, S_out), -7, dtype=torch.int32, device=dev)
        fm.Coords2TypedCoords_forward(rows(x), rows(rn), rows(an), rows(na), out, cnt, off, idx)
        assert fm.workspace_status(0) == 0
        assert torch.equal(cnt, rows(wcnt)) and torch.equal(off, rows(woff))
        assert torch.equal(out[:, :3 * wide], rows(want)) and not out[:, 3 * wide:].any()
        assert torch.equal(idx[:, :wide], rows(widx).to(torch.int32)) and not idx[:, wide:].any()
        if S == 33:
            bad = an.copy()
            bad[1, 4] = list(b"QQ\0\0")
            out.fill_(float("nan"))
            fm.Coords2TypedCoords_forward(rows(x), rows(rn), rows(bad), rows(na), out, cnt, off, idx)
            assert fm.workspace_status(0) != 0
            assert int(cnt[1].sum()) == int(na[1]) - 1 and int(cnt[0].sum()) == 0 and torch.isfinite(out).all()
