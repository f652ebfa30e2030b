"""Tile ids 9-12 run the kernels of ids 0 and 2-4, so no model may tell them apart: equal predictions, choices
that fall on the first name, and training rows of both names that count for one kernel.  The C++ chooser maps
the same ids."""
import math
import re

from conftest import ROOT
from mgxbench_b200 import autotune as at

PAIRS = [(0, 9), (2, 10), (3, 11), (4, 12)]


def test_features_and_regression_see_one_kernel():
    assert sorted((b, a) for a, b in at.SAME_KERNEL.items()) == PAIRS
    for a, b in PAIRS:
        ca, cb = at.Candidate(a, 0), at.Candidate(b, 0)
        assert ca.ksplit == cb.ksplit and at.features(300, 400, 5000, 7, ca) == at.features(300, 400, 5000, 7, cb)
    rows = [{"m": n, "n": n, "k": n, "exp_range": 0, "tile": t, "splits": 0, "seconds": s * n ** 3 * 1e-13, "error": 1e-16}
            for n in (300, 900, 2700) for t, s in ((0, 1.0), (9, 1.21), (13, 1.05))]
    reg = at.RegressionModel().fit(rows)
    cs = [at.Candidate(t, 0) for t in (13, 0, 9)]
    (sk, _), (whole, _), (alias, _) = reg.predict(1000, 1000, 1000, 0, cs)
    assert whole == alias and math.isclose(whole, 1.1e-4, rel_tol=1e-9) and math.isclose(sk, 1.05e-4, rel_tol=1e-9)
    assert at.choose(reg, 1000, 1000, 1000, 0, 1e-15, cs[1:]).tile == 0


def test_cpp_chooser_maps_the_same_ids():
    text = (ROOT / "mgxbench_b200" / "host" / "autotune.h").read_text()
    body = text[text.index("inline int model_tile"):]
    got = re.findall(r"case (\d+): return (\d+);", body[:body.index("}\n}")])
    assert sorted((int(b), int(a)) for a, b in got) == PAIRS
    assert re.search(r"feat\[6\] = \{[^}]*model_tile\(\(int\)cand\[2 \* c\]\)", text)


def test_packaged_sweep_is_of_these_kernels():
    """Both names of a kernel were measured alike, and the packaged network was trained on the packaged sweep."""
    import json
    import statistics
    db = at.SweepDB(ROOT / "mgxbench_b200" / "data" / "sweep_b200.jsonl")
    held = {}
    for r in db.rows:
        if r.get("set") == "heldout":
            held.setdefault((r["m"], r["n"], r["k"], r["exp_range"]), {})[(r["tile"], r["splits"])] = r["seconds"]
    for a, b in PAIRS:
        ratios = [abs(math.log(d[a, 0] / d[b, 0])) for d in held.values() if (a, 0) in d and (b, 0) in d]
        assert len(ratios) > 300 and statistics.quantiles(ratios, n=10)[-1] < 0.1
    model = json.loads((ROOT / "mgxbench_b200" / "data" / "mlp_b200.json").read_text())
    assert model["training_set"] == db.digest()
