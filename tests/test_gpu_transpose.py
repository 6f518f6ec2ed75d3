"""The transposes between layouts (GPU): pixels, channels and strides around the 4 x 4 elements of a lane and the 32 x
128 of a block, with and without 16-byte alignment; and the lines-fastest products at every line count of their vector
loads, all angles at once and a list of angles in several chunks, from a buffer that is not 16-byte aligned, and with
more blocks than four waves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("npix,K,k0,kb,kstride", [(1, 3, 1, 2, 8), (4, 8, 0, 8, 8), (31, 9, 2, 7, 8), (64, 40, 4, 33, 40),
                                                  (9801, 20, 3, 17, 24), (1028, 300, 0, 300, 304), (130, 129, 1, 128, 128)])
@pytest.mark.parametrize("shift", [0, 1])
def test_gather_and_scatter_channels(npix, K, k0, kb, kstride, shift):
    from diffractom_b200 import _lib
    s = torch.cuda.current_stream().cuda_stream
    flat = torch.randn(K * npix + shift, device="cuda")
    x = flat[shift:].view(K, npix)                     # shift 1: not 16-byte aligned
    img = torch.full((npix, kstride), 7.0, device="cuda")
    _lib.call("dfx_gather_channels", x.data_ptr(), img.data_ptr(), npix, k0, kb, kstride, s)
    want = torch.zeros((npix, kstride), device="cuda")
    want[:, :kb] = x[k0:k0 + kb].t()
    assert torch.equal(img, want)
    src = torch.randn((npix, kstride), device="cuda")
    out = torch.full((K * npix + shift,), 7.0, device="cuda")
    y = out[shift:].view(K, npix)
    _lib.call("dfx_scatter_channels", src.data_ptr(), y.data_ptr(), npix, k0, kb, kstride, s)
    want = torch.full((K, npix), 7.0, device="cuda")
    want[k0:k0 + kb] = src[:, :kb].t()
    assert torch.equal(y, want) and (out[:shift] == 7.0).all()


def _rows(rng, n, width, max_len):
    lens = rng.integers(0, max_len + 1, n)
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = np.concatenate([np.sort(rng.choice(width, m, replace=False)) for m in lens] + [np.zeros(1)]).astype(np.uint16)
    return ptr, idx


def _products(my, listed, shift, chunk):
    """Random block rows and adjoint rows of R angles; runs both lines-fastest products (angles in `listed`, None: all;
    a buffer of `chunk` angles, `shift` floats off) and returns (inputs, forward data, adjoint rows)."""
    from diffractom_b200 import _lib
    rng = np.random.default_rng(my)
    P, C, R, kb, ks = 3, 9, 5, 50, 56
    cp, ncb = P * C, 3
    dev = lambda a: torch.as_tensor(a, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    ptr, fk = _rows(rng, R * P * ncb, kb, 21)
    fv = rng.standard_normal((len(fk), 4)).astype(np.float32)
    mask = np.full((R, ncb, P), 15, np.uint8)
    mask[:, -1] = 1                                    # the last eta block has one bin
    n = R if listed is None else len(listed)
    om = None if listed is None else dev(np.asarray(listed, np.int32))
    omp = None if om is None else om.data_ptr()
    sino = rng.standard_normal((n, my, ks)).astype(np.float32)
    data = rng.standard_normal((R, my, cp)).astype(np.float32)
    aptr, col = _rows(rng, R * kb, cp, 19)
    val = rng.standard_normal(len(col)).astype(np.float32)
    d = [dev(v) for v in (ptr, fk.view(np.int16), fv, mask.reshape(-1), sino, data, aptr, col.view(np.int16), val)]
    lib = _lib.lib()
    ly = -(-my // 32) * 32
    floats = (lib.dfx_spmm_pf_forward_zt_floats(chunk, my, kb), lib.dfx_spmm_pf_adjoint_zt_floats(chunk, my, cp))
    assert floats == (chunk * kb * ly, chunk * cp * ly)
    zt = torch.empty(max(floats) + 4, device="cuda")[shift:]
    fwd, adj = d[5].clone(), torch.full((n, my, ks), 5.0, device="cuda")
    _lib.call("dfx_spmm_pf_forward_blocked_zt", d[4].data_ptr(), zt.data_ptr(), floats[0], *(v.data_ptr() for v in d[:4]),
              fwd.data_ptr(), omp, n, my, P, C, ks, kb, 0, s)
    _lib.call("dfx_spmm_pf_adjoint_zt", d[5].data_ptr(), zt.data_ptr(), floats[1], *(v.data_ptr() for v in d[6:]),
              adj.data_ptr(), omp, n, my, kb, cp, ks, 1.5, 0, 0, s)
    return (P, C, R, kb, ks, ncb, om, d, (ptr, fk, fv, sino, data, aptr, col, val)), fwd, adj


@pytest.mark.parametrize("my", [1, 32, 33, 64, 90, 128, 129, 190, 224, 256, 257, 289, 330])
@pytest.mark.parametrize("listed,chunk", [(None, 5), ([3, 0, 4], 2)])
def test_lines_fastest_products_at_every_line_count(my, listed, chunk):
    """Both products against their channel-fastest forms, bit for bit; a list of angles goes through a buffer of two."""
    from diffractom_b200 import _lib
    (P, C, R, kb, ks, ncb, om, d, _), fwd, adj = _products(my, listed, 0, chunk)
    s = torch.cuda.current_stream().cuda_stream
    n, omp = adj.shape[0], None if om is None else om.data_ptr()
    a, b = d[5].clone(), torch.full_like(adj, 5.0)
    _lib.call("dfx_spmm_pf_forward_blocked", d[4].data_ptr(), *(v.data_ptr() for v in d[:4]), a.data_ptr(), omp, n, my, P,
              C, ks, kb, s)
    assert torch.equal(a, fwd) and not torch.equal(a, d[5])
    _lib.call("dfx_spmm_pf_adjoint", d[5].data_ptr(), *(v.data_ptr() for v in d[6:]), b.data_ptr(), omp, n, my, kb, P * C,
              ks, 1.5, 0, s)
    assert torch.equal(b, adj) and b[:, :, :kb].any() and not b[:, :, kb:].any()


@pytest.mark.parametrize("shift", [0, 1])
def test_lines_fastest_products_against_float64(shift):
    """Both products within one float32 rounding per term and one per addition; shift 1: a buffer that is not 16-byte
    aligned."""
    my, listed = 70, [3, 0, 4]
    (P, C, R, kb, ks, ncb, om, d, (ptr, fk, fv, sino, data, aptr, col, val)), fwd, adj = _products(my, listed, shift, 2)
    want, size = data.astype(np.float64), np.abs(data).astype(np.float64)
    wadj, sadj = np.zeros((3, my, kb)), np.zeros((3, my, kb))
    for i, r in enumerate(listed):
        for g in range(P * ncb):
            cb, p = divmod(g, P)
            e = slice(ptr[r * P * ncb + g], ptr[r * P * ncb + g + 1])
            for u in range(min(4, C - 4 * cb)):
                t = sino[i][:, fk[e]].astype(np.float64) * fv[e, u]
                want[r, :, (4 * cb + u) * P + p] += t.sum(1)
                size[r, :, (4 * cb + u) * P + p] += np.abs(t).sum(1)
        for k in range(kb):
            e = slice(aptr[r * kb + k], aptr[r * kb + k + 1])
            t = 1.5 * data[r][:, col[e]].astype(np.float64) * val[e]
            wadj[i, :, k], sadj[i, :, k] = t.sum(1), np.abs(t).sum(1)
    assert (np.abs(fwd.cpu().numpy() - want) <= 24 * 2.0 ** -24 * size).all()
    assert (np.abs(adj.cpu().numpy()[:, :, :kb] - wadj) <= 24 * 2.0 ** -24 * sadj).all()


@pytest.mark.parametrize("my", [20, 53, 70, 263])
def test_lines_fastest_forward_with_many_blocks(my):
    """Many blocks (the variants with three of them per SM): the channel-fastest form's bits."""
    from diffractom_b200 import _lib
    rng = np.random.default_rng(7)
    P, C, R, kb, ks = 8, 36, 400, 40, 40               # 400 angles x 5 blocks of two eta blocks
    ncb = 9
    dev = lambda a: torch.as_tensor(a, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    ptr, fk = _rows(rng, R * P * ncb, kb, 9)
    fv = dev(rng.standard_normal((len(fk), 4)).astype(np.float32))
    mask = torch.full((R * P * ncb,), 15, dtype=torch.uint8, device="cuda")
    ptr, fk = dev(ptr), dev(fk.view(np.int16))
    sino = dev(rng.standard_normal((R, my, ks)).astype(np.float32))
    a = torch.zeros((R, my, P * C), device="cuda")
    b = torch.zeros_like(a)
    zt = torch.empty(_lib.lib().dfx_spmm_pf_forward_zt_floats(R, my, kb), device="cuda")
    _lib.call("dfx_spmm_pf_forward_blocked", sino.data_ptr(), ptr.data_ptr(), fk.data_ptr(), fv.data_ptr(),
              mask.data_ptr(), a.data_ptr(), None, R, my, P, C, ks, kb, s)
    _lib.call("dfx_spmm_pf_forward_blocked_zt", sino.data_ptr(), zt.data_ptr(), zt.numel(), ptr.data_ptr(), fk.data_ptr(),
              fv.data_ptr(), mask.data_ptr(), b.data_ptr(), None, R, my, P, C, ks, kb, 0, s)
    assert torch.equal(a, b) and a.any()
