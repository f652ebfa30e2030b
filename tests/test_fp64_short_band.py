"""CPU restatement of the FP64 kernel's work cut where the last band has one or two 16-row strips and its
units cost less (launch_dgemm, Walk, sk_start and sk_unit in csrc/fp64_gemm.cu): the CTAs' shares cover
every unit once, in order and evenly by cost; the warps of a tile cover its strips and units once; the
piece index and partial slot of a stream-K segment are the ones the finishing warp looks up."""
import pytest

TILE_UNITS, BM, COST, COSTS, CWARPS = 16, 64, 8, {1: 3, 2: 5}, 16


def cut(m, n):
    bands, ucols = -(-m // BM), -(-n // 8)
    tiles_n = -(-ucols // TILE_UNITS)
    return bands, ucols, -(-ucols // tiles_n), tiles_n


def weights(m, n, kblocks, grid, sms, streamk, slices=1):
    """(strips of the last band, cost of a unit, cost of a unit of the last band)"""
    bands, ucols, _, tiles_n = cut(m, n)
    strips = -(-(m - (bands - 1) * BM) // 16)
    if strips > 2:
        return 4, 1, 1
    w, row = COSTS[strips], tiles_n * kblocks
    if bands == 1:
        return strips, 1, 1
    weigh = row * ((bands - 1) * COST + w) >= grid * COST if streamk else bands * ucols * slices > sms
    return (strips, COST, w) if weigh else (4 if streamk else strips, 1, 1)


def sk_begin(c, U, G):
    return c * U // G


def sk_owner(u, U, G):
    return ((u + 1) * G + U - 1) // U - 1


SHAPES = [(1, 1), (16, 9), (32, 4096), (65, 129), (80, 512), (96, 4096), (257, 257), (272, 1024), (777, 1281),
          (1040, 4096), (130, 260), (4097, 40), (16, 8192), (2080, 2048)]


@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("slices", [1, 3])
@pytest.mark.parametrize("sms", [148, 7, 1])
def test_shares_cover_the_product_once_and_evenly(m, n, slices, sms):
    bands, ucols, _, _ = cut(m, n)
    units = bands * ucols * slices
    G = min(units, sms)
    skew = 2 if units >= 8 * G else 0
    strips, wf, wl = weights(m, n, 1, G, sms, False, slices)
    row_len, slice_len = (ucols + skew) * wf, (bands - 1) * (ucols + skew) * wf + skew * wf + ucols * wl

    def row_unit(pos):
        sl, pos = divmod(pos, slice_len)
        band = min(pos // row_len, bands - 1)
        w = wl if band == bands - 1 else wf
        off = pos - band * row_len - skew * wf
        return (sl * bands + band) * ucols + (0 if off <= 0 else -(-off // w))

    U, end, load = slices * slice_len, 0, []
    for c in range(G):
        x, x_end = row_unit(sk_begin(c, U, G)), row_unit(sk_begin(c + 1, U, G))
        assert x == end and x_end >= x
        end = x_end
        load.append(sum(wl if (u // ucols) % bands == bands - 1 else wf for u in range(x, x_end)))
    assert end == units
    assert max(load) < U // G + 1 + wf


@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("kblocks", [1, 2, 33, 188])
@pytest.mark.parametrize("sms", [148, 7])
def test_stream_k_pieces(m, n, kblocks, sms):
    bands, _, _, tiles_n = cut(m, n)
    tiles = bands * tiles_n
    G = min(tiles * kblocks, sms)
    strips, wf, wl = weights(m, n, kblocks, G, sms, True)
    full = (bands - 1 if wl < wf else bands) * tiles_n * kblocks

    def start(x):
        return x * wf if x < full else full * wf + (x - full) * wl

    def unit(pos):
        rest = pos - full * wf
        return -(-pos // wf) if rest <= 0 else full + -(-rest // wl)

    U, end, seen = start(tiles * kblocks), 0, {}
    for c in range(G):
        x, x_end = unit(sk_begin(c, U, G)), unit(sk_begin(c + 1, U, G))
        assert x == end and x_end > x
        end = x_end
        while x < x_end:
            t = x // kblocks
            k0, k1 = x - t * kblocks, min(kblocks, x - t * kblocks + x_end - x)
            c0 = sk_owner(start(t * kblocks), U, G)
            pieces = sk_owner(start(t * kblocks + kblocks - 1), U, G) - c0 + 1
            slot = 0 if x == unit(sk_begin(c, U, G)) else 1
            j = c - c0
            assert slot == ((0 if unit(sk_begin(c0, U, G)) == t * kblocks else 1) if j == 0 else 0)
            seen.setdefault(t, []).append((k0, k1, j, pieces))
            x += k1 - k0
    assert end == tiles * kblocks
    for segs in seen.values():
        assert [s[2] for s in segs] == list(range(segs[0][3])) and segs[0][0] == 0 and segs[-1][1] == kblocks
        assert all(a[1] == b[0] for a, b in zip(segs, segs[1:]))


@pytest.mark.parametrize("strips", [1, 2, 4])
@pytest.mark.parametrize("units", range(1, TILE_UNITS + 1))
def test_warps_cover_a_tile_once(strips, units):
    sharers = CWARPS // strips
    per = -(-units // sharers)
    got = []
    for cw in range(CWARPS):
        first = cw // strips * per
        got += [(cw & (strips - 1), u) for u in range(first, first + max(0, min(per, units - first)))]
    assert per <= 4 and sorted(got) == [(s, u) for s in range(strips) for u in range(units)]
