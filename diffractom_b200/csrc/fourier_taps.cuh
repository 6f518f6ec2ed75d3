// Index arithmetic of the Fourier-slice spread (fourier.cu), in plain C++ so that a host program can replay it over an
// angle set's tables (tests/test_fourier.py): taps have offsets 0 .. W-1, on cells of the half grid only.
#pragma once

#ifdef __CUDACC__
#define FR_HD __host__ __device__ __forceinline__
#else
#define FR_HD inline
#endif

namespace dfx {

constexpr int FR_TS = 16;     // spreading tile (cells per side)

FR_HD int wrap(int v, int m)
{
    const int r = v % m;
    return r < 0 ? r + m : r;
}

// The first tap of a sample along one axis of m cells as the spread stages it: b, or -b through the mirror, modulo m.
FR_HD int fr_first(int b, bool mir, int m) { return wrap(mir ? -b : b, m); }

// Offset of cell q from a staged first tap: q - b, through the mirror b - q, wrapped once. In 0 .. m-1 for cells of the
// axis (0 <= q < m); for FR_OFF and the cells after it either negative or far above W.
FR_HD int fr_offset(int q, int b, bool mir, int m)
{
    const int d = mir ? b - q : q - b;
    return d < 0 ? d + m : d;
}

constexpr int FR_OFF = 1 << 30;

// Cell q of an axis of m cells, FR_OFF if a tile reaches past the axis there: without it the offset of a mirrored sample
// can be negative, and the offsets of both kinds can pass for taps.
FR_HD int fr_cell(int q, int m) { return q < m ? q : FR_OFF; }

// Does a sample have a tap on cell q (fr_cell) of an axis, at offset d?
FR_HD bool fr_tap(int q, int b, bool mir, int m, int W, int &d)
{
    d = fr_offset(q, b, mir, m);
    return (unsigned)d < (unsigned)W;
}

// Does a sample have a tap on row0 (fr_cell) or the row after it? (A row past an odd axis may say yes: its cells find no
// tap.)
FR_HD bool fr_rows_near(int row0, int b2, bool mir, int My, int W)
{
    int d;
    return fr_tap(row0, b2, mir, My, W, d) || fr_tap(row0 + 1, b2, mir, My, W, d);
}

}  // namespace dfx
