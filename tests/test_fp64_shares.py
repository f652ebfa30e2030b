"""CPU restatement of the FP64 kernel's work cut (Walk and dgemm_cut in csrc/fp64_gemm.cu): equal
shares of the 8-column units of all (band, K slice) rows.  The CTAs' pieces must cover every
(band, unit, K slice) exactly once, in pieces no wider than a tile, and load the CTAs equally."""
import pytest

TILE_UNITS = 16


def pieces(c, G, bands, slices, ucols, skew):
    row_len = ucols + skew
    U = bands * slices * row_len
    u, u_end = c * U // G, (c + 1) * U // G
    while u < u_end:
        row = u // row_len
        off = u - row * row_len - skew
        if off < 0:
            u -= off
            off = 0
            if u >= u_end:
                return
        run = min(ucols - off, u_end - u)
        width = -(-run // -(-run // TILE_UNITS))
        u += width
        yield row % bands, row // bands, off, width


@pytest.mark.parametrize("m,n,slices", [(1, 1, 1), (64, 8, 1), (65, 129, 1), (256, 256, 1), (1024, 1024, 1),
                                        (777, 1281, 3), (3001, 5002, 1), (1000, 9000, 1), (130, 260, 16),
                                        (16384, 129, 1), (16384, 8, 1), (2200, 72, 1)])
@pytest.mark.parametrize("sms", [148, 7, 1])
def test_shares_cover_the_product_once_and_evenly(m, n, slices, sms):
    bands, ucols = -(-m // 64), -(-n // 8)
    units = bands * ucols * slices
    G = min(sms, units)
    skew = 2 if units >= 8 * G else 0
    seen, load = set(), []
    for c in range(G):
        total = 0
        for band, sl, u0, width in pieces(c, G, bands, slices, ucols, skew):
            assert 0 <= band < bands and 0 <= sl < slices and 1 <= width <= TILE_UNITS and u0 + width <= ucols
            for u in range(u0, u0 + width):
                assert (band, sl, u) not in seen
                seen.add((band, sl, u))
            total += width
        load.append(total)
    assert len(seen) == units
    assert max(load) <= -(-bands * slices * (ucols + skew) // G)
