"""The native projector's kernels at the sizes where their work split can go wrong (GPU): channel counts around the 256
of a warp and its two runs of 128, bins around the groups of four, angle counts around a block's, image widths around a
tile's, detectors narrower than the image (taps at its edge), both footprints."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (nx, ny, bins, angles, kb, kstride)
SIZES = [(5, 4, 6, 3, 1, 8), (8, 7, 9, 9, 12, 16), (17, 21, 11, 13, 127, 128), (19, 16, 24, 8, 130, 136),
         (33, 30, 41, 17, 250, 256), (16, 18, 15, 16, 257, 264), (23, 9, 26, 7, 500, 504), (12, 35, 37, 5, 1000, 1008)]
# the backprojection's four-pixel rows serve images of 3552 (BF16 rows), 4144 or 4736 (with the primal step) pixels x 256
# channels on: sizes on both sides of those lines (one and two channel groups), widths around a row's four pixels,
# detectors narrower than the image
LARGE = [(73, 65, 60, 3, 1, 8), (74, 64, 79, 9, 250, 256), (37, 128, 120, 8, 256, 256), (47, 50, 44, 17, 257, 264),
         (49, 49, 55, 7, 500, 504), (131, 75, 90, 5, 127, 128), (56, 74, 70, 6, 129, 136), (53, 67, 60, 11, 30, 32),
         (41, 51, 48, 10, 300, 304)]


def _geometry(nx, ny, bins, angles, kernel):
    from diffractom_b200.geometry import radon_geometry
    ang = (np.arange(angles) + 0.5) * np.pi / angles
    return radon_geometry(ang, nx, ny, bins, float(max(nx, ny)), float(bins), 0.3, np.pi / angles, kernel)


def _tables(rg, nx, ny, bins, kid, group):
    from diffractom_b200 import _lib
    s = torch.cuda.current_stream().cuda_stream
    geo = torch.as_tensor(rg.geo, device="cuda")
    R = len(rg.geo)
    kind = "gtable" if group else "table"
    cnt = torch.empty(R * (-(-bins // 4) if group else bins), dtype=torch.int32, device="cuda")
    _lib.call(f"dfx_radon_{kind}_count", geo.data_ptr(), R, nx, ny, bins, kid, None, cnt.data_ptr(), s)
    rp = torch.zeros(cnt.numel() + 1, dtype=torch.int32, device="cuda")
    rp[1:] = cnt.cumsum(0)
    n = max(int(rp[-1].item()), 1)
    if not group:
        ent = torch.empty(2 * n, dtype=torch.int32, device="cuda")
        _lib.call("dfx_radon_table_fill", geo.data_ptr(), R, nx, ny, bins, kid, None, rp.data_ptr(), ent.data_ptr(), s)
        return rp, ent
    pix, w = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty((n, 4), device="cuda")
    _lib.call("dfx_radon_gtable_fill", geo.data_ptr(), R, nx, ny, bins, kid, None, rp.data_ptr(), pix.data_ptr(),
              w.data_ptr(), s)
    return rp, pix, w


@pytest.mark.parametrize("kernel", ["trapezoid", "hat"])
@pytest.mark.parametrize("size", SIZES, ids=str)
def test_forward_tables_equal_the_footprint_forward(size, kernel):
    """Per-bin and grouped table forwards, float32 and BF16 rows, all angles and a list: dfx_radon_forward's bits
    (the BF16 rows its values rounded once); padding channels are not read."""
    from diffractom_b200 import _lib
    nx, ny, bins, R, kb, ks = size
    rg = _geometry(nx, ny, bins, R, kernel)
    kid, scale, s = int(kernel == "trapezoid"), float(rg.scale), torch.cuda.current_stream().cuda_stream
    geo = torch.as_tensor(rg.geo, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(3)
    img = torch.randn((nx * ny, ks), generator=g, device="cuda")
    img[:, kb:] = float("nan")
    ref = torch.empty((R, bins, ks), device="cuda")
    _lib.call("dfx_radon_forward", img.data_ptr(), ref.data_ptr(), geo.data_ptr(), R, nx, ny, bins, ks, kb, kid, scale, s)
    assert torch.isfinite(ref).all() and not ref[:, :, kb:].any()
    rp, ent = _tables(rg, nx, ny, bins, kid, False)
    grp = _tables(rg, nx, ny, bins, kid, True)
    some = torch.arange(R - 1, -1, -2, dtype=torch.int32, device="cuda")
    ld = ks + 8
    for om in (None, some):
        n = R if om is None else om.numel()
        want = ref if om is None else ref[om.long()]
        op = None if om is None else om.data_ptr()
        out, outb = torch.empty((n, bins, ks), device="cuda"), torch.empty((n, bins, ld), dtype=torch.bfloat16, device="cuda")
        _lib.call("dfx_radon_forward_table", img.data_ptr(), out.data_ptr(), rp.data_ptr(), ent.data_ptr(), op, n, bins,
                  ks, kb, scale, s)
        assert torch.equal(out, want)
        _lib.call("dfx_radon_forward_table_bf16", img.data_ptr(), outb.data_ptr(), ld, rp.data_ptr(), ent.data_ptr(), op,
                  n, bins, ks, kb, scale, s)
        assert torch.equal(outb[:, :, :ks], want.to(torch.bfloat16))
        out.zero_(), outb.zero_()
        _lib.call("dfx_radon_forward_gtable", img.data_ptr(), out.data_ptr(), *(t.data_ptr() for t in grp), op, n, bins,
                  ks, kb, scale, s)
        assert torch.equal(out, want)
        _lib.call("dfx_radon_forward_gtable_bf16", img.data_ptr(), outb.data_ptr(), ld, *(t.data_ptr() for t in grp), op,
                  n, bins, ks, kb, scale, s)
        assert torch.equal(outb[:, :, :ks], want.to(torch.bfloat16))


def test_bf16_image_table_forward_equals_the_float32_one():
    """A BF16 image (widened exactly) through the per-bin table: the float32 forward of the same values."""
    from diffractom_b200 import _lib
    for nx, ny, bins, R, kb, ks in SIZES:
        rg = _geometry(nx, ny, bins, R, "trapezoid")
        s = torch.cuda.current_stream().cuda_stream
        g = torch.Generator(device="cuda").manual_seed(4)
        img = torch.randn((nx * ny, ks), generator=g, device="cuda").to(torch.bfloat16)
        img32 = img.float()
        rp, ent = _tables(rg, nx, ny, bins, 1, False)
        a = torch.empty((R, bins, ks), dtype=torch.bfloat16, device="cuda")
        b = torch.empty_like(a)
        _lib.call("dfx_radon_forward_table_bf16_bf16", img.data_ptr(), a.data_ptr(), ks, rp.data_ptr(), ent.data_ptr(),
                  None, R, bins, ks, kb, float(rg.scale), s)
        _lib.call("dfx_radon_forward_table_bf16", img32.data_ptr(), b.data_ptr(), ks, rp.data_ptr(), ent.data_ptr(), None,
                  R, bins, ks, kb, float(rg.scale), s)
        assert torch.equal(a, b)


@pytest.mark.parametrize("kernel", ["trapezoid", "hat"])
@pytest.mark.parametrize("size", SIZES + LARGE, ids=str)
def test_backprojection_of_whole_images_equals_the_pixel_lists(size, kernel):
    """dfx_radon_backward (rows of pixels sharing bins from a few thousand warps on) = dfx_radon_backward_pixels over
    every pixel (pixel by pixel, two channel groups per warp from as many warps on) and over a row of pixels, bit for
    bit: float32 and BF16 rows with their own stride, padding channels 0; dfx_radon_backward_spdhg = the backprojection
    followed by dfx_spdhg_primal_update, the padding channels of x, z kept."""
    from diffractom_b200 import _lib
    nx, ny, bins, R, kb, ks = size
    rg = _geometry(nx, ny, bins, R, kernel)
    kid, nt, s = int(kernel == "trapezoid"), int(rg.n_taps), torch.cuda.current_stream().cuda_stream
    assert nt == 2
    geo = torch.as_tensor(rg.geo, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(5)
    sino = torch.randn((R, bins, ks), generator=g, device="cuda")
    pix = torch.arange(nx * ny, dtype=torch.int32, device="cuda")
    want, out = torch.empty((nx * ny, ks), device="cuda"), torch.empty((nx * ny, ks), device="cuda")

    def pixels(src):
        _lib.call("dfx_radon_backward_pixels", src.data_ptr(), want.data_ptr(), geo.data_ptr(), R, nx, ny, bins, ks, kb,
                  kid, nt, pix.data_ptr(), nx * ny, s)

    pixels(sino)
    _lib.call("dfx_radon_backward", sino.data_ptr(), out.data_ptr(), geo.data_ptr(), R, nx, ny, bins, ks, kb, kid, nt, s)
    assert torch.equal(out, want) and want.any() and not want[:, kb:].any()
    row = torch.empty((nx, ks), device="cuda")         # a launch of few warps whatever the image
    _lib.call("dfx_radon_backward_pixels", sino.data_ptr(), row.data_ptr(), geo.data_ptr(), R, nx, ny, bins, ks, kb, kid,
              nt, pix[(ny // 2) * nx:].data_ptr(), nx, s)
    assert torch.equal(row, want[(ny // 2) * nx:(ny // 2 + 1) * nx])
    # the primal step in the epilogue
    x, z, T = (torch.rand((nx * ny, ks), generator=g, device="cuda") for _ in range(3))
    x[:, kb:] = z[:, kb:] = T[:, kb:] = 0
    xr, zr = x.clone(), z.clone()
    _lib.call("dfx_spdhg_primal_update", xr.data_ptr(), zr.data_ptr(), T.data_ptr(), want.data_ptr(), 7.0, 0.25,
              x.numel(), s)
    _lib.call("dfx_radon_backward_spdhg", sino.data_ptr(), geo.data_ptr(), R, nx, ny, bins, ks, kb, kid, nt, x.data_ptr(),
              z.data_ptr(), T.data_ptr(), 7.0, 0.25, s)
    assert torch.equal(x, xr) and torch.equal(z, zr)
    # BF16 rows of a wider sinogram
    ld = ks + 8
    sb = torch.randn((R, bins, ld), generator=g, device="cuda").to(torch.bfloat16)
    pixels(sb[:, :, :ks].float().contiguous())
    _lib.call("dfx_radon_backward_bf16", sb.data_ptr(), ld, out.data_ptr(), geo.data_ptr(), R, nx, ny, bins, ks, kb, kid,
              nt, s)
    assert torch.equal(out, want)


def test_backprojection_with_more_than_two_taps():
    """Pixels wider than the bins (three or four taps a pixel): the general kernel, against the forward's transpose
    in float64 (2 x 20 angles x 4 taps of float32 rounding)."""
    from diffractom_b200 import _lib
    from diffractom_b200.geometry import radon_geometry
    nx, ny, bins, R, kb, ks = 9, 11, 31, 20, 40, 48
    ang = (np.arange(R) + 0.5) * np.pi / R
    rg = radon_geometry(ang, nx, ny, bins, 28.0, float(bins), 0.0, 1.0, "trapezoid")
    assert rg.n_taps > 2
    s = torch.cuda.current_stream().cuda_stream
    geo = torch.as_tensor(rg.geo, device="cuda")
    eye = torch.zeros((nx * ny, 104), device="cuda")
    eye[torch.arange(nx * ny), torch.arange(nx * ny)] = 1.0
    A = torch.empty((R, bins, 104), device="cuda")
    _lib.call("dfx_radon_forward", eye.data_ptr(), A.data_ptr(), geo.data_ptr(), R, nx, ny, bins, 104, 104, 1, 1.0, s)
    sino = torch.randn((R, bins, ks), device="cuda")
    out = torch.empty((nx * ny, ks), device="cuda")
    _lib.call("dfx_radon_backward", sino.data_ptr(), out.data_ptr(), geo.data_ptr(), R, nx, ny, bins, ks, kb, 1,
              int(rg.n_taps), s)
    want = torch.einsum("abp,abk->pk", A[:, :, :nx * ny].double(), sino.double())
    bound = torch.einsum("abp,abk->pk", A[:, :, :nx * ny].double().abs(), sino.double().abs()) * 2 * R * 4 * 2.0 ** -24
    assert ((out.double() - want).abs()[:, :kb] <= bound[:, :kb]).all() and not out[:, kb:].any()


@pytest.mark.parametrize("bins,width,taps", [(150, 140.0, 3), (301, 280.0, 5), (90, 140.0, 3)])
@pytest.mark.parametrize("ks,kb", [(304, 300), (8, 5)])
def test_more_than_two_taps_two_at_a_time(bins, width, taps, ks, kb):
    """Three to five taps a pixel, detectors wider and narrower than the image: a row of pixels (few warps, the taps'
    rows loaded in pairs) = the same pixels of the whole image (two channel groups per warp at 304 channels) bit for
    bit, float32 and BF16 rows (widened exactly); and the float64 sum of the oracle's weights within its rounding."""
    from diffractom_b200 import _lib
    from diffractom_b200.geometry import radon_geometry
    nx, ny, R = 70, 40, 13
    ang = (np.arange(R) + 0.5) * np.pi / R
    rg = radon_geometry(ang, nx, ny, bins, width, float(bins), 0.3, 0.7, "trapezoid")
    assert rg.n_taps == taps
    s = torch.cuda.current_stream().cuda_stream
    geo = torch.as_tensor(rg.geo, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(8)
    sino = torch.randn((R, bins, ks), generator=g, device="cuda").to(torch.bfloat16).float()
    full, fullb, row = (torch.empty((n, ks), device="cuda") for n in (nx * ny, nx * ny, nx))
    _lib.call("dfx_radon_backward", sino.data_ptr(), full.data_ptr(), geo.data_ptr(), R, nx, ny, bins, ks, kb, 1, taps, s)
    sb = sino.to(torch.bfloat16)
    _lib.call("dfx_radon_backward_bf16", sb.data_ptr(), ks, fullb.data_ptr(), geo.data_ptr(), R, nx, ny, bins, ks, kb, 1,
              taps, s)
    assert torch.equal(full, fullb) and full.any() and not full[:, kb:].any()
    for y in (0, 17, ny - 1):
        pix = torch.arange(y * nx, (y + 1) * nx, dtype=torch.int32, device="cuda")
        _lib.call("dfx_radon_backward_pixels", sino.data_ptr(), row.data_ptr(), geo.data_ptr(), R, nx, ny, bins, ks, kb, 1,
                  taps, pix.data_ptr(), nx, s)
        assert torch.equal(row, full[y * nx:(y + 1) * nx])
    # float64: the trapezoid of a unit step along the axis with the larger coefficient
    geo64 = np.asarray(rg.geo, np.float64)
    yy, xx = (v.ravel() for v in np.mgrid[:ny, :nx])
    want, size = np.zeros((nx * ny, kb)), np.zeros((nx * ny, kb))
    src = sino[:, :, :kb].double().cpu().numpy()
    for a in range(R):
        t = geo64[a, 0] * xx + geo64[a, 1] * yy + geo64[a, 2]
        A = max(abs(geo64[a, 0]), abs(geo64[a, 1]))
        w = np.clip((1 + A) / 2 - np.abs(t[:, None] - np.arange(bins)), 0.0, min(1.0, A)) / A * geo64[a, 3]
        want += w @ src[a]
        size += w @ np.abs(src[a])
    # the place of a pixel is rounded to 2^-24 of some hundred bins, a weight's slope is 1 / A, 5 taps of each angle
    bound = 2 * R * taps * 2.0 ** -24 * size + 2.0 ** -24 * bins * 4 * np.abs(src).max() * R * 0.7 * taps
    assert (np.abs(full[:, :kb].double().cpu().numpy() - want) <= bound).all()
