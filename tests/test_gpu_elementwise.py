"""Element-wise kernels with a vector and a general form (GPU): both forms at lengths and alignments around the vector's,
against torch."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _s():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("n", [1, 3, 4, 7, 1000, 70001])
@pytest.mark.parametrize("grad", [0, 1])
def test_poisson_value_and_gradient_of_plain_counts(n, grad):
    """The deviance sum in float64 to n roundings of its terms' absolute sum; the gradient, and with it the form with
    unaligned arrays (the general kernel), to one float32 rounding of the float64 value."""
    from diffractom_b200 import _lib
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(n)
    mu0 = torch.randn(n, generator=g, device="cuda") * 3 + 4
    b = torch.poisson(torch.full((n,), 4.0, device="cuda"), generator=g)
    b[::5] = 0
    eps = 1e-3
    m = mu0.clamp_min(0).double() + float(torch.tensor(eps, dtype=torch.float32))
    bd = b.double()
    terms = m - bd + torch.where(b > 0, bd * torch.log(torch.where(b > 0, bd, torch.ones_like(bd)) / m), torch.zeros_like(m))
    want = 1 - bd / m
    scr = torch.empty(lib.dfx_reduce_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    for shift in (0, 1):
        buf, cnt = torch.empty(n + 1, device="cuda")[shift:shift + n], torch.empty(n + 1, device="cuda")[shift:shift + n]
        buf.copy_(mu0), cnt.copy_(b)
        _lib.call("dfx_poisson_value_grad", buf.data_ptr(), cnt.data_ptr(), None, 0, None, 0, None, 0, eps, grad, 0, 0.0, n,
                  out.data_ptr(), scr.data_ptr(), scr.numel(), _s())
        # a term's own rounding is that of bd log(bd / m), a few ulp of |bd| and m
        bound = (n + 16) * 2.0 ** -53 * float((m + 4 * bd + terms.abs()).sum())
        assert abs(float(out) - float(terms.sum())) <= bound
        if grad:
            assert ((buf.double() - want).abs() <= want.abs() * 2.0 ** -23 + 1e-14).all()
        else:
            assert torch.equal(buf, mu0)


@pytest.mark.parametrize("npix,ks,kb,shift", [(1, 8, 3, 0), (37, 16, 13, 0), (64, 1008, 1000, 0), (9, 5, 4, 0), (21, 8, 8, 1)])
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("masked", [False, True])
def test_batch_support(npix, ks, kb, shift, mode, masked):
    from diffractom_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(npix)
    x0 = torch.randn((npix, ks), generator=g, device="cuda")
    cs = torch.randn((npix, ks), generator=g, device="cuda")
    supp = (torch.rand(npix, generator=g, device="cuda") < 0.6).to(torch.uint8) if masked else None
    flat = torch.empty(npix * ks + 1, device="cuda")[shift:shift + npix * ks]
    flat.copy_(x0.reshape(-1))
    inside = torch.zeros((npix, ks), dtype=torch.bool, device="cuda")
    inside[:, :kb] = True
    if masked:
        inside &= supp.bool()[:, None]
    zero = torch.zeros_like(x0)
    want = {0: inside.float(), 1: torch.where(inside & ~(x0 < 0), x0, zero),
            2: torch.where(inside & (cs > 0), torch.minimum(x0, 0.7 / cs), x0), 3: torch.where(inside, x0, zero)}[mode]
    _lib.call("dfx_batch_support", flat.data_ptr(), cs.data_ptr(), None if supp is None else supp.data_ptr(), npix, ks, kb,
              0.7, mode, _s())
    assert torch.allclose(flat.view(npix, ks), want, rtol=2.0 ** -22, atol=0)


@pytest.mark.parametrize("R,my,cp,pad,shift", [(3, 5, 16, 16, 0), (4, 7, 24, 24, 0), (2, 3, 13, 16, 0), (3, 1, 8, 8, 1),
                                               (2, 263, 2880, 2880, 0), (2, 19, 127, 128, 0), (2, 9, 129, 136, 0)])
def test_rows_to_bf16(R, my, cp, pad, shift):
    from diffractom_b200 import _lib
    x = torch.empty(R * my * cp + 1, device="cuda")[shift:shift + R * my * cp].view(R, my, cp)
    x.copy_(torch.randn((R, my, cp), device="cuda"))
    for om in (None, torch.tensor([R - 1, 0], dtype=torch.int32, device="cuda")):
        out = torch.full((R, my, pad), 9.0, dtype=torch.bfloat16, device="cuda")
        rows = range(R) if om is None else om.tolist()
        _lib.call("dfx_rows_to_bf16", x.data_ptr(), out.data_ptr(), None if om is None else om.data_ptr(), len(rows), my, cp,
                  pad, _s())
        for r in range(R):
            if r in rows:
                assert torch.equal(out[r, :, :cp], x[r].to(torch.bfloat16)) and not out[r, :, cp:].any()
            else:
                assert (out[r] == 9.0).all()
