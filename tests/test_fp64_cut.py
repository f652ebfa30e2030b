"""The FP64 kernel's work cut as it ships: csrc/fp64_cut.h compiled for the host.  The CTAs' shares cover every
unit of work once, in order and evenly by cost; a stream-K segment's piece and slot are the ones that the
finishing warp looks up; the warps cover a tile's strips and units once; positions fit 32 bits."""
import ctypes
import subprocess

import numpy as np
import pytest

from conftest import ROOT

WHOLE, PANELS, STREAMK = 0, 1, 2

HARNESS = r"""
#include "fp64_cut.h"
using namespace mgx::fp64;

extern "C" {

// cut: bands, ucols, tile_units, tiles_n, kblocks, skew, strips_last, w_full, w_last, grid; returns the length
long long cut_of(int m, int n, int k, int ksplit, int kb_split, int mode, int sms, int *cut)
{
    int grid = 0;
    const Cut p = make_cut(m, n, k, ksplit, kb_split, (CutMode)mode, sms, &grid);
    const int v[10] = {p.bands, p.ucols, p.tile_units, p.tiles_n, p.kblocks, p.skew, p.strips_last, p.w_full, p.w_last, grid};
    for (int i = 0; i < 10; ++i) cut[i] = v[i];
    return p.length;
}

// the first units of every CTA's share and the end of the last
void shares(int m, int n, int k, int ksplit, int kb_split, int mode, int sms, long long *x)
{
    int grid = 0;
    const Cut p = make_cut(m, n, k, ksplit, kb_split, (CutMode)mode, sms, &grid);
    for (int c = 0; c < grid; ++c) {
        if (mode == 2) {
            Walk<true, long long> w;
            w.init(p, c, grid);
            x[c] = w.x;
            x[c + 1] = w.x_end;
        } else {
            Walk<false, unsigned> w;
            w.init(p, c, grid);
            if (c > 0 && x[c] != (long long)w.x) x[c] = -1;
            else x[c] = w.x;
            x[c + 1] = w.x_end;
        }
    }
}

// every item of every CTA: cta, band, u0, units, kb_begin, kb_end, slice, strips, tile, c0, pieces, index, slot, slot0
int items(int m, int n, int k, int ksplit, int kb_split, int mode, int sms, int *out, int room)
{
    int grid = 0, count = 0;
    const Cut p = make_cut(m, n, k, ksplit, kb_split, (CutMode)mode, sms, &grid);
    auto put = [&](int c, const Item &it, const Piece &q) {
        const int v[14] = {c, it.band, it.u0, it.units, it.kb_begin, it.kb_end, it.slice, it.strips, it.tile,
                           q.c0, q.pieces, q.index, q.slot, q.slot0};
        if (count < room)
            for (int i = 0; i < 14; ++i) out[14 * count + i] = v[i];
        ++count;
    };
    for (int c = 0; c < grid; ++c) {
        Item it = {};
        if (mode == 2) {
            Walk<true, long long> w;
            w.init(p, c, grid);
            while (w.next(p, it)) put(c, it, piece_of(p, it, c, grid));
        } else {
            Walk<false, unsigned> w;
            w.init(p, c, grid);
            while (w.next(p, it)) put(c, it, Piece{});
        }
    }
    return count;
}

void warps(int units, int strips, int *out)
{
    Item it = {};
    it.units = units;
    it.strips = strips;
    for (int cw = 0; cw < CWARPS; ++cw) warp_part(it, cw, out[3 * cw], out[3 * cw + 1], out[3 * cw + 2]);
}

int constants(int i) { const int v[3] = {BM, TILE_UNITS, CWARPS}; return v[i]; }
}
"""


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    d = tmp_path_factory.mktemp("cut")
    (d / "cut.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wno-unknown-pragmas", "-shared", "-fPIC", "-fsanitize=undefined",
                    "-fno-sanitize-recover=undefined", "-static-libubsan", "-I", str(ROOT / "mgxbench_b200" / "csrc"),
                    "-o", str(d / "cut.so"), str(d / "cut.cpp")], check=True)
    L = ctypes.CDLL(str(d / "cut.so"))
    L.cut_of.restype = ctypes.c_longlong
    return L


def slices(k, asked):
    kblocks = -(-k // 32)
    kb_split = -(-kblocks // min(max(asked, 1), kblocks))
    return -(-kblocks // kb_split), kb_split


def load(L, m, n, k, asked, mode, sms):
    ks, kb = slices(k, asked)
    v = (ctypes.c_int * 10)()
    length = L.cut_of(m, n, k, ks, kb, mode, sms, v)
    names = ("bands", "ucols", "tile_units", "tiles_n", "kblocks", "skew", "strips_last", "w_full", "w_last", "grid")
    c = dict(zip(names, v), length=length, ksplit=ks, kb_split=kb)
    room = L.items(m, n, k, ks, kb, mode, sms, None, 0)
    buf = np.zeros((max(room, 1), 14), np.int32)
    L.items(m, n, k, ks, kb, mode, sms, buf.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), room)
    return c, buf[:room]


SHAPES = [(1, 1), (64, 8), (65, 129), (256, 256), (1024, 1024), (777, 1281), (3001, 5002), (1000, 9000), (130, 260),
          (16384, 129), (16384, 8), (2200, 72), (16, 9), (32, 4096), (80, 512), (272, 1024), (1040, 4096), (4097, 40),
          (2080, 2048), (9472, 16)]


@pytest.mark.parametrize("m,n", SHAPES)
def test_shares_cover_the_product_once_and_evenly(cut, m, n):
    for mode, asked in ((WHOLE, 1), (WHOLE, 3), (WHOLE, 16), (PANELS, 1)):
        for sms in (148, 7, 1):
            check_shares(cut, m, n, asked, mode, sms)


def check_shares(cut, m, n, asked, mode, sms):
    c, it = load(cut, m, n, 1000, asked, mode, sms)
    bm, tile_units = cut.constants(0), cut.constants(1)
    assert c["bands"] == -(-m // bm) and c["ucols"] == -(-n // 8) and c["grid"] <= sms
    seen = np.zeros((c["ksplit"], c["bands"], c["ucols"]), np.int32)
    cost = np.zeros(c["grid"])
    order = -1
    for (cta, band, u0, units, kb0, kb1, sl, strips, *_) in it:
        assert 1 <= units <= tile_units and kb0 == sl * c["kb_split"] and kb1 == min(c["kblocks"], kb0 + c["kb_split"])
        seen[sl, band, u0:u0 + units] += 1
        at = (sl * c["bands"] + band) * c["ucols"] + u0
        assert at > order and u0 + units <= c["ucols"]
        order = at
        last = band == c["bands"] - 1
        assert strips == (c["strips_last"] if last else 2)
        # the strips that are computed hold all of the band's rows
        assert 16 << strips >= min(bm, m - band * bm)
        cost[cta] += units * (c["w_last"] if last else c["w_full"])
    assert (seen == 1).all()
    assert mode == WHOLE or c["strips_last"] == 2
    # no share is longer than its part of the length, the unit that begins at its end included
    assert cost.max() < c["length"] // c["grid"] + 1 + c["w_full"]


@pytest.mark.parametrize("m,n", SHAPES)
def test_stream_k_pieces(cut, m, n):
    for k in (1, 33, 1056, 6001):
        for sms in (148, 7, 1, 300):
            check_pieces(cut, m, n, k, sms)


def check_pieces(cut, m, n, k, sms):
    c, it = load(cut, m, n, k, 1, STREAMK, sms)
    tiles, kblocks = c["bands"] * c["tiles_n"], c["kblocks"]
    assert len(set(it[:, 0])) == c["grid"]          # every CTA has a unit: it is counted among a tile's pieces
    by_tile, corner = {}, set()
    for (cta, band, u0, units, kb0, kb1, sl, strips, tile, c0, pieces, index, slot, slot0) in it:
        assert 0 <= kb0 < kb1 <= kblocks and cta == c0 + index and slot in (0, 1)
        # the finishing warp's lookup: the first piece in slot0 of CTA c0, the others in slot 0
        assert pieces == 1 or slot == (slot0 if index == 0 else 0)
        by_tile.setdefault(tile, []).append((kb0, kb1, index, pieces))
        corner.add((tile, band, u0, units, strips))
    assert sorted(by_tile) == list(range(tiles)) and len(corner) == tiles
    # a short last band is weighed only where shares hold four whole units
    assert c["w_last"] == c["w_full"] == 1 or c["length"] >= 4 * c["w_full"] * c["grid"]
    cover = np.zeros((c["bands"], c["ucols"]), np.int32)
    for (_, band, u0, units, strips) in corner:
        cover[band, u0:u0 + units] += 1
        assert 16 << strips >= min(64, m - band * 64)
    assert (cover == 1).all()
    for segs in by_tile.values():
        assert [s[2] for s in segs] == list(range(len(segs))) and all(s[3] == len(segs) for s in segs)
        assert segs[0][0] == 0 and segs[-1][1] == kblocks and all(a[1] == b[0] for a, b in zip(segs, segs[1:]))


@pytest.mark.parametrize("strips", [0, 1, 2])
def test_warps_cover_a_tile_once(cut, strips):
    n = cut.constants(2)
    out = (ctypes.c_int * (3 * n))()
    for units in range(1, 17):
        cut.warps(units, strips, out)
        got = [(out[3 * w], u) for w in range(n) for u in range(out[3 * w + 1], out[3 * w + 1] + out[3 * w + 2])]
        assert max(out[3 * w + 2] for w in range(n)) <= 4
        assert sorted(got) == [(s, u) for s in range(1 << strips) for u in range(units)]


# (2^31 - 1) x 1 in 20 slices of an even pitch is more than a B200 holds, and 24 units of cost a band
@pytest.mark.parametrize("m,n,k,asked", [(2 ** 31 - 1, 1, 32, 1), (2 ** 31 - 63, 9, 32, 1), (2 ** 31 - 63, 1, 700, 20),
                                         (2 ** 31 - 63, 3, 3200, 100), (2 ** 30 + 1, 17, 1280, 40), (1, 2 ** 31 - 1, 32, 1)])
@pytest.mark.parametrize("mode", [WHOLE, PANELS])
def test_positions_fit_32_bits(cut, m, n, k, asked, mode):
    asked = asked if mode == WHOLE else 1
    ks, kb = slices(k, asked)
    v = (ctypes.c_int * 10)()
    length = cut.cut_of(m, n, k, ks, kb, mode, 148, v)
    assert 0 < length < 2 ** 32
    x = (ctypes.c_longlong * (v[9] + 1))()
    cut.shares(m, n, k, ks, kb, mode, 148, x)
    units = v[0] * v[1] * ks
    assert v[0] == -(-m // 64) and v[1] == -(-n // 8)
    assert x[0] == 0 and x[v[9]] == units and all(0 <= a <= b for a, b in zip(x, x[1:]))
    # even by count where every unit costs the same
    if v[7] == v[8]:
        assert max(b - a for a, b in zip(x, x[1:])) <= length // v[9] + 1
