"""CPU restatement of the CRT form's residue arithmetic (all_residues in csrc/ozaki_crt.cu), with its
table of modulus pairs read from the source: the FP32 stage over every value the FP64 stage can leave,
and the FP64 stage against exact integers."""
import random
import re
from fractions import Fraction

import numpy as np
import pytest

from conftest import ROOT

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193]
ROUND = 6755399441055744


def pair_sets():
    text = (ROOT / "mgxbench_b200" / "csrc" / "ozaki_crt.cu").read_text()
    body = text[text.index("constexpr PairSet kPairs"):]
    body = body[:body.index("};\n")]
    sets = {}
    for q, pairs, single in re.findall(r"/\* +(\d+) \*/ \{\{(.*?)\}, (-?\d+)\}", body):
        sets[int(q)] = ([tuple(map(int, t)) for t in re.findall(r"\{(\d+), (\d+), (\d+)\}", pairs)], int(single))
    return sets


def offset(pp, M):
    bits = 0x4B000000 + M - 2 ** 23
    odd, target, mod = (pp // 256, -(bits // 256), 2 ** 24) if pp % 2 == 0 else (pp, -bits, 2 ** 32)
    return target * pow(odd, -1, mod) % mod


def symmetric(z, p):
    return (z + p // 2) % p - p // 2


def test_every_modulus_is_paired_once():
    sets = pair_sets()
    assert sorted(sets) == list(range(8, 17))
    for q, (pairs, single) in sets.items():
        used = [i for a, b, _ in pairs for i in (a, b)] + ([single] if single >= 0 else [])
        assert sorted(used) == list(range(q))
        for a, b, M in pairs:
            pp = MODULI[a] * MODULI[b]
            assert M % 256 == 0 and 2 ** 23 + pp + 4 < M < 2 ** 24 - pp - 4
            assert (pp * offset(pp, M) + 0x4B000000 + M - 2 ** 23) % 2 ** 32 == 0


@pytest.mark.parametrize("pair", sorted({p for pairs, _ in pair_sets().values() for p in pairs}))
def test_second_stage_for_every_z(pair):
    a, b, M = pair
    lim = MODULI[a] * MODULI[b] + 4
    z = np.arange(-lim, lim + 1, dtype=np.int64)
    u = 0x4B000000 + (M - 2 ** 23) + z
    assert np.array_equal(u.astype(np.uint32).view(np.float32).astype(np.float64), (M + z).astype(np.float64))
    for p in (MODULI[a], MODULI[b]):
        ip = np.float64(np.float32(1.0 / p))
        c = 12582912.0 - np.floor(M * ip + 0.5)
        assert np.float64(np.float32(c)) == c
        t = ((M + z) * ip + c).astype(np.float32).view(np.int32).astype(np.int64)   # one FP32 rounding
        assert np.array_equal((u - t * p) & 255, symmetric(z, p) & 255)


@pytest.mark.parametrize("q", range(8, 17))
def test_first_stage_against_integers(q):
    rng = random.Random(q)
    pairs, single = pair_sets()[q]
    xs = [0, 1, -1, 2 ** 31, -2 ** 31, 2 ** 32, 2 ** 62, -2 ** 62, 2 ** 63 - 2 ** 10, -2 ** 63 + 2 ** 10]
    for _ in range(400):
        e = rng.randrange(0, 63)
        x = rng.randrange(-2 ** e, 2 ** e + 1)
        xs.append(int(float(x)))          # the scaled value is a double
    for x in xs:
        xh = int(round(Fraction(x, 2 ** 32)))   # nearest, ties to even
        xl = x - xh * 2 ** 32
        assert abs(xl) <= 2 ** 31 and abs(xh) <= 2 ** 31
        for a, b, M in pairs:
            pp = MODULI[a] * MODULI[b]
            y = xh * (2 ** 32 % pp) + xl
            ip = Fraction(1.0 / pp)
            magic = ROUND + offset(pp, M) - int(float(ROUND) * (1.0 / pp) + 0.5)
            t = int(round((ROUND + y) * ip + magic))
            assert 2 ** 52 <= t < 2 ** 53 and abs(y) < 2 ** 50
            u = (y - pp * t) % 2 ** 32          # low words: 1.5 * 2^52 is a multiple of 2^32
            z = u - (0x4B000000 + M - 2 ** 23)
            assert abs(z) <= pp + 4 and (z - x) % pp == 0
        if single >= 0:
            p = MODULI[single]
            y = xh * (2 ** 32 % p) + xl
            t = int(round(y * Fraction(1.0 / p)))
            assert y - p * t == symmetric(x, p)
