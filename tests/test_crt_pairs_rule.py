"""The CRT form's rule for pairs of CTAs, csrc/crt_pairs.h compiled for the host: never more pairs than can be
resident at once (the rest would start after the others, which wait for them at every item), and only
where their rounds of items are no more than single CTAs'."""
import ctypes
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs")
    (d / "pairs.cpp").write_text('#include "crt_pairs.h"\nextern "C" int rule(long long items, long long pairs, int sms, '
                                 'int clusters) { return mgx::crt::pairs_to_launch(items, pairs, sms, clusters); }\n')
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-shared", "-fPIC", "-I", str(ROOT / "mgxbench_b200" / "csrc"),
                    "-o", str(d / "pairs.so"), str(d / "pairs.cpp")], check=True)
    L = ctypes.CDLL(str(d / "pairs.so"))
    L.rule.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    return L.rule


@pytest.mark.parametrize("sms,clusters", [(148, 74), (148, 60), (148, 1), (148, 0), (132, 66), (1, 0), (7, 3)])
def test_no_more_pairs_than_are_resident(rule, sms, clusters):
    for tiles_m in (1, 2, 3, 9, 16, 64):
        for tiles_n in (1, 5, 8, 64):
            for q in (8, 15):
                items, pairs = q * tiles_m * tiles_n, q * ((tiles_m + 1) // 2) * tiles_n
                n = rule(items, pairs, sms, clusters)
                assert 0 <= n <= min(clusters, sms // 2)
                if n:
                    assert pairs >= 4 * n and -(-pairs // n) <= -(-items // sms)


def test_whole_gpu(rule):
    assert rule(15 * 64 * 64, 15 * 32 * 64, 148, 74) == 74     # 16384^3
    assert rule(15 * 6 * 8, 15 * 3 * 8, 148, 74) == 74         # 1333 x 2011: 5 rounds of either
    assert rule(15 * 4 * 4, 15 * 2 * 4, 148, 74) == 0          # 1024^3: 2 rounds
    assert rule(15 * 5 * 16, 15 * 3 * 16, 148, 74) == 0        # an odd last tile row: 10 rounds against 9
