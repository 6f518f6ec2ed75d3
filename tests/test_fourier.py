"""The Fourier-slice projector's host tables on the CPU: a NumPy run of the device pipeline (pad, 2-D FFT,
interpolation, 1-D inverse FFT; and the transposed steps with the spreading tile lists) built from the same float32
tables matches the exact Fourier-slice projection of the oracle to the NUFFT's accuracy, and the exact projection
agrees with the native (hat) projector to the few per cent that separate the two projectors."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from diffractom_b200.fourier import FourierHost
from oracle import fourier as orc

GEOMS = [dict(Nx=22, Ny=18, Ns=30, R=11, shift=0.35, width=22.0), dict(Nx=16, Ny=16, Ns=17, R=7, shift=0.0, width=16.0)]


def _host(g, arc=np.pi):
    ang = np.linspace(0, arc, g["R"], endpoint=False) + 0.021
    h = FourierHost(ang, g["Nx"], g["Ny"], g["Ns"], g["width"], float(g["Ns"]), g["shift"], np.pi / g["R"])
    return h, ang


def _emulated_forward(h, tab, img):
    """img (Ny, Nx, C) -> sino (R, Ns, C) through the tables (float64 arithmetic)."""
    C = img.shape[-1]
    grid = np.zeros((C, h.My, h.Mx))
    for y in range(h.Ny):
        for x in range(h.Nx):
            grid[:, (y - h.cy) % h.My, (x - h.cx) % h.Mx] = img[y, x] * h.inv_dx[x] * h.inv_dy[y]
    G = np.fft.fft2(grid)                                     # the full (Hermitian) spectrum
    W = h.W
    taps = np.arange(W)
    k1 = (tab.kb[:, 0, None] + taps) % h.Mx                  # (RH, W)
    k2 = (tab.kb[:, 1, None] + taps) % h.My
    w = tab.w2.astype(np.float64)[:, :, None] * tab.w1.astype(np.float64)[:, None, :]     # (RH, l, i)
    vals = G[:, k2[:, :, None], k1[:, None, :]]               # (C, RH, l, i)
    acc = (vals * w[None]).sum(axis=(2, 3))
    spec = acc * tab.filt.astype(np.complex128)[None]
    j = np.arange(tab.RH) % tab.H
    spec[:, (j == 0) | (j == tab.H - 1)] = spec[:, (j == 0) | (j == tab.H - 1)].real
    lines = np.fft.irfft(spec.reshape(C, tab.R, tab.H), n=h.L, axis=-1) * h.L
    return (float(h.scale) * lines[:, :, :h.Ns]).transpose(1, 2, 0)


def _emulated_backward(h, tab, sino):
    """sino (R, Ns, C) -> img (Ny, Nx, C) through the tables and the spreading tile lists."""
    R, Ns, C = sino.shape
    lines = np.zeros((C, R, h.L))
    lines[:, :, :Ns] = (sino * tab.wa.astype(np.float64)[:, None, None]).transpose(2, 0, 1)
    spec = np.fft.rfft(lines, axis=-1).reshape(C, tab.RH) * np.conj(tab.filt.astype(np.complex128))[None]
    Hx = h.Mx // 2 + 1
    Q = np.zeros((C, h.My, Hx), complex)
    TS = 16
    for tile in range(tab.n_tiles):
        q1 = (tile % tab.n_tx) * TS + np.arange(TS)[None, :]
        q2 = (tile // tab.n_tx) * TS + np.arange(TS)[:, None]
        inside = (q1 < Hx) & (q2 < h.My)
        for e in range(tab.tile_ptr[tile], tab.tile_ptr[tile + 1]):
            sm = int(tab.tile_smp[e])
            mir, smp = sm < 0, (sm if sm >= 0 else -sm - 1)
            p1, p2 = (-q1, -q2) if mir else (q1, q2)
            d1 = (p1 - tab.kb[smp, 0]) % h.Mx
            d2 = (p2 - tab.kb[smp, 1]) % h.My
            hit = inside & (d1 < h.W) & (d2 < h.W)
            if not hit.any():
                continue
            j = smp % tab.H
            half = 0.5 if j in (0, tab.H - 1) else 1.0
            wgt = tab.w2[smp, np.minimum(d2, h.W - 1)].astype(np.float64) * tab.w1[smp, np.minimum(d1, h.W - 1)] * half
            v = np.conj(spec[:, smp]) if mir else spec[:, smp]
            qq2, qq1 = np.nonzero(hit)
            Q[:, q2[qq2, 0], q1[0, qq1]] += wgt[hit][None, :] * v[:, None]
    grid = np.fft.irfft2(Q, s=(h.My, h.Mx)) * (h.My * h.Mx)
    img = np.zeros((h.Ny, h.Nx, C))
    for y in range(h.Ny):
        for x in range(h.Nx):
            img[y, x] = grid[:, (y - h.cy) % h.My, (x - h.cx) % h.Mx] * h.inv_dx[x] * h.inv_dy[y]
    return img


@pytest.mark.parametrize("g", GEOMS)
def test_tables_reproduce_the_exact_fourier_slice_projection(g):
    h, ang = _host(g)
    tab = h.tables()
    M, scale, L = orc.fourier_slice_matrix(ang, g["Nx"], g["Ny"], g["Ns"], g["width"], float(g["Ns"]), g["shift"])
    assert L == h.L and scale == float(h.scale)
    rng = np.random.default_rng(1)
    img = rng.random((g["Ny"], g["Nx"], 3))
    ref = orc.forward(M, scale, img.reshape(-1, 3))
    out = _emulated_forward(h, tab, img)
    assert np.abs(out - ref).max() <= 1e-4 * np.abs(ref).max()
    sino = rng.standard_normal((g["R"], g["Ns"], 2))
    refb = orc.backward(M, np.pi / g["R"], sino).reshape(g["Ny"], g["Nx"], 2)
    outb = _emulated_backward(h, tab, sino)
    assert np.abs(outb - refb).max() <= 1e-4 * np.abs(refb).max()


def test_subset_tables_are_the_rows_of_their_angles():
    g = GEOMS[0]
    h, ang = _host(g)
    full, sub = h.tables(), h.tables(np.arange(2, g["R"], 3))
    rows = np.concatenate([np.arange(a * full.H, (a + 1) * full.H) for a in range(2, g["R"], 3)])
    assert np.array_equal(sub.kb, full.kb[rows]) and np.array_equal(sub.w1, full.w1[rows])
    assert np.array_equal(sub.filt, full.filt[rows]) and np.array_equal(sub.wa, full.wa[2::3])


def test_exact_projection_is_close_to_the_native_hat_projector():
    """The Fourier-slice projector band-limits the bin's hat; on a smooth image it agrees with the native hat
    projector to a few per cent in norm (the reference documents about 1 % on reconstructions); pointwise the
    native projector's aliasing at some angles makes the difference larger."""
    g = dict(Nx=32, Ny=32, Ns=46, R=12, shift=0.0, width=32.0)
    h, ang = _host(g)
    M, scale, _ = orc.fourier_slice_matrix(ang, g["Nx"], g["Ny"], g["Ns"], g["width"], float(g["Ns"]))
    yy, xx = np.mgrid[:32, :32]
    img = np.exp(-((xx - 15.3) ** 2 + (yy - 16.8) ** 2) / 40.0).ravel()
    fs = orc.forward(M, scale, img[:, None])[..., 0]
    X, Y, T = h.XYT_all
    t = X[:, None] * (xx.ravel() - h.cx)[None] + Y[:, None] * (yy.ravel() - h.cy)[None] + T[:, None]
    d = np.arange(g["Ns"])[None, :, None] - t[:, None, :]
    hat = np.maximum(0.0, 1.0 - np.abs(d))
    native = scale * (hat * img[None, None, :]).sum(-1)
    rel = np.linalg.norm(fs - native) / np.linalg.norm(native)
    assert rel <= 0.03, rel


def test_spreading_pieces_partition_every_tile_list():
    """Every tile's sample list is cut into pieces in order (at most PIECE samples each); a tile's first piece has
    no slot, its later pieces the consecutive slots tile_xptr[t] ..; empty lists keep one (empty) piece."""
    from diffractom_b200.fourier import PIECE
    g = dict(Nx=64, Ny=60, Ns=90, R=90, shift=0.1, width=64.0)
    h, _ = _host(g)
    tab = h.tables()
    pc = tab.pieces
    assert np.diff(tab.tile_ptr).max() > PIECE                    # some lists need several pieces
    for t in range(tab.n_tiles):
        mine = pc[pc[:, 0] == t]
        assert mine[0, 1] == tab.tile_ptr[t] and mine[-1, 2] == tab.tile_ptr[t + 1]
        assert np.array_equal(mine[1:, 1], mine[:-1, 2]) and np.all(mine[:, 2] - mine[:, 1] <= PIECE)
        assert mine[0, 3] == -1 and np.array_equal(mine[1:, 3], np.arange(tab.tile_xptr[t], tab.tile_xptr[t + 1]))
    assert tab.n_slots == len(pc) - tab.n_tiles


REPLAY = r"""
#include "fourier_taps.cuh"
#include <cstdint>
using namespace dfx;
// out[entry][thread] = d2 W + d1 of the tap that the spread's thread applies for the tile list's entry, -1: none
extern "C" void replay(const int32_t *tile_ptr, const int32_t *tile_smp, const int32_t *kb, int n_tiles, int n_tx,
                       int Mx, int My, int W, int32_t *out)
{
    for (int tile = 0; tile < n_tiles; ++tile)
        for (int e = tile_ptr[tile]; e < tile_ptr[tile + 1]; ++e) {
            const int sm = tile_smp[e], smp = sm >= 0 ? sm : -sm - 1;
            const bool mir = sm < 0;
            const int b1 = fr_first(kb[2 * smp], mir, Mx), b2 = fr_first(kb[2 * smp + 1], mir, My);
            for (int lid = 0; lid < FR_TS * FR_TS; ++lid) {
                const int lx = lid % FR_TS, ly = lid / FR_TS;
                const int q1 = fr_cell(tile % n_tx * FR_TS + lx, Mx / 2 + 1), q2 = fr_cell(tile / n_tx * FR_TS + ly, My);
                int d1, d2, &o = out[(int64_t)e * FR_TS * FR_TS + lid] = -1;
                if (!fr_rows_near(fr_cell(tile / n_tx * FR_TS + (ly & ~1), My), b2, mir, My, W)) continue;
                if (fr_tap(q1, b1, mir, Mx, W, d1) && fr_tap(q2, b2, mir, My, W, d2))
                    o = d1 >= 0 && d2 >= 0 && d1 < W && d2 < W ? d2 * W + d1 : -2;
            }
        }
}
"""


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    """The spread's index arithmetic (csrc/fourier_taps.cuh) compiled for the host."""
    d = tmp_path_factory.mktemp("replay")
    (d / "replay.cpp").write_text(REPLAY)
    inc = Path(__file__).resolve().parents[1] / "diffractom_b200" / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(inc), str(d / "replay.cpp"), "-o",
                    str(d / "replay.so")], check=True)
    return ctypes.CDLL(str(d / "replay.so")).replay


@pytest.mark.parametrize("W", [6, 7])
@pytest.mark.parametrize("Nx,Ny,R", [(416, 416, 5), (100, 100, 24), (64, 70, 24), (128, 128, 9), (5, 7, 9), (9, 4, 7)])
def test_spread_reads_only_taps_of_cells_on_the_grid(replay, Nx, Ny, R, W):
    """The taps that the spread's threads apply, replayed on the host over the tables: exactly those of the cells on the
    half grid, by modular arithmetic; none on a tile's rows or columns past it (grids whose sides are no multiple of the
    tile's, and narrower than a tile). An offset outside 0 .. W-1 would read past the staged weights."""
    ang = np.linspace(0, np.pi, R, endpoint=False) + 0.021
    h = FourierHost(ang, Nx, Ny, max(Nx, Ny) + 3, float(max(Nx, Ny)), max(Nx, Ny) + 3.0, 0.2, np.pi / R, W=W)
    tab = h.tables()
    n = len(tab.tile_smp)
    got = np.empty((n, 16, 16), np.int32)
    arr = [np.ascontiguousarray(a, np.int32) for a in (tab.tile_ptr, tab.tile_smp, tab.kb)]
    replay(*(a.ctypes.data_as(ctypes.c_void_p) for a in arr), tab.n_tiles, tab.n_tx, h.Mx, h.My, W,
           got.ctypes.data_as(ctypes.c_void_p))
    tile = np.repeat(np.arange(tab.n_tiles), np.diff(tab.tile_ptr))
    mir = tab.tile_smp < 0
    smp = np.where(mir, -tab.tile_smp - 1, tab.tile_smp)
    sign = np.where(mir, -1, 1)[:, None]
    q1 = (tile % tab.n_tx * 16)[:, None] + np.arange(16)
    q2 = (tile // tab.n_tx * 16)[:, None] + np.arange(16)
    d1 = ((sign * q1 - tab.kb[smp, :1]) % h.Mx)[:, None, :]
    d2 = ((sign * q2 - tab.kb[smp, 1:]) % h.My)[:, :, None]
    inside = (q1 <= h.Mx // 2)[:, None, :] & (q2 < h.My)[:, :, None]
    want = np.where(inside & (d1 < W) & (d2 < W), d2 * W + d1, -1)
    assert np.array_equal(got, want) and (want >= 0).any()
