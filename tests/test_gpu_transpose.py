"""The transposes between layouts (GPU): pixels, channels and strides around the 4 x 4 elements of a lane and the 32 x
128 of a block, with and without 16-byte alignment; and the lines-fastest products at every line count of their vector
loads, from a buffer that is not 16-byte aligned, and with more blocks than four waves."""
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


@pytest.mark.parametrize("my", [1, 32, 33, 64, 90, 128, 129, 190, 224, 256, 257, 289, 330])
@pytest.mark.parametrize("shift", [0, 1])
def test_lines_fastest_products_at_every_line_count(my, shift):
    """Both products against their channel-fastest forms, bit for bit; shift 1: the buffer is not 16-byte aligned."""
    from diffractom_b200 import _lib
    rng = np.random.default_rng(my)
    P, C, R, kb, ks = 3, 9, 3, 50, 56
    cp, ncb = P * C, 3
    dev = lambda a: torch.as_tensor(a, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    ptr, fk = _rows(rng, R * P * ncb, kb, 21)
    fv = dev(rng.standard_normal((len(fk), 4)).astype(np.float32))
    mask = dev(np.full(R * P * ncb, 15, np.uint8).reshape(R, ncb, P))
    mask[:, -1] = 1                                    # the last eta block has one bin
    ptr, fk = dev(ptr), dev(fk.view(np.int16))
    sino = dev(rng.standard_normal((R, my, ks)).astype(np.float32))
    data = dev(rng.standard_normal((R, my, cp)).astype(np.float32))
    a, b = data.clone(), data.clone()
    lib = _lib.lib()
    zt = torch.empty(max(lib.dfx_spmm_pf_forward_zt_floats(R, my, kb), lib.dfx_spmm_pf_adjoint_zt_floats(R, my, cp)) + 4,
                     device="cuda")[shift:]
    _lib.call("dfx_spmm_pf_forward_blocked", sino.data_ptr(), ptr.data_ptr(), fk.data_ptr(), fv.data_ptr(),
              mask.data_ptr(), a.data_ptr(), None, R, my, P, C, ks, kb, s)
    _lib.call("dfx_spmm_pf_forward_blocked_zt", sino.data_ptr(), zt.data_ptr(), zt.numel(), ptr.data_ptr(), fk.data_ptr(),
              fv.data_ptr(), mask.data_ptr(), b.data_ptr(), None, R, my, P, C, ks, kb, 0, s)
    assert torch.equal(a, b) and not torch.equal(a, data)
    ptr, col = (dev(v) for v in _rows(rng, R * kb, cp, 19))
    val = dev(rng.standard_normal(col.numel()).astype(np.float32))
    col = col.view(torch.int16)
    a, b = (torch.full((R, my, ks), 5.0, device="cuda") for _ in range(2))
    _lib.call("dfx_spmm_pf_adjoint", data.data_ptr(), ptr.data_ptr(), col.data_ptr(), val.data_ptr(), a.data_ptr(), None, R,
              my, kb, cp, ks, 1.5, 0, s)
    _lib.call("dfx_spmm_pf_adjoint_zt", data.data_ptr(), zt.data_ptr(), zt.numel(), ptr.data_ptr(), col.data_ptr(),
              val.data_ptr(), b.data_ptr(), None, R, my, kb, cp, ks, 1.5, 0, 0, s)
    assert torch.equal(a, b) and a[:, :, :kb].any() and not a[:, :, kb:].any()


@pytest.mark.parametrize("my", [70, 263])
def test_lines_fastest_forward_with_many_blocks(my):
    """More than four waves of blocks (the variant with three blocks per SM): the channel-fastest form's bits."""
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
