"""Workloads of this library as its users run them, with inputs, one pass through the public entry
points, the work a pass cannot do without, and its results in plain 64-bit torch.

A case is a dict of plain values: `kind` says which entry points a pass calls, the other keys are
sizes and options of those calls.

  fp64       one native FP64 product: `ab_multiply` (the reference's call), or `gemm_fp64` with the
             K-slice and tile options that the autotuner offers
  rows       a 1D row-block run: one FP64 product per emulated rank's row block
  chunks     one rank of the K-chunked 1D pipeline: C = 0, then C += A[:, chunk] B_chunk
  summa      a 2D SUMMA plan over an uneven process grid
  ozaki      the INT8 digit-slice form
  crt        the INT8 residue (CRT) form
  host       a product of host buffers, copies overlapped with the product
  validate   the reference's constant check of a whole C
  mlp        one training step of the autotuner's cost model, then its prediction
"""
from __future__ import annotations

import math

import torch

import mgxbench_b200 as mgx

CHUNK = 2048          # the 1D pipeline's default K chunk
PANEL = 256           # the SUMMA drivers' default panel width
FORMS = {"fp64": mgx.FORM_FP64, "ozaki": mgx.FORM_OZAKI, "crt": mgx.FORM_CRT}


def listed():
    return [
        # the smallest product that a benchmark sweep starts with: launches and latency
        {"name": "fp64_n256", "kind": "fp64", "m": 256, "n": 256, "k": 256, "odd": False, "call": "ab"},
        # the reference's plain product at N = 1024, one 1D block
        {"name": "fp64_n1024", "kind": "fp64", "m": 1024, "n": 1024, "k": 1024, "odd": False, "call": "ab"},
        # N = 8192 over 4 ranks: 2048 x 8192 row blocks in sequence
        {"name": "fp64_rows_n8192", "kind": "rows", "n": 8192, "ranks": 4},
        # one of 4 ranks of the K-chunked pipeline at N = 4096, default chunk
        {"name": "fp64_chunks_n4096", "kind": "chunks", "m": 1024, "n": 4096, "k": 4096, "chunk": CHUNK},
        # ragged block with odd pitches, few output tiles and a long K: the autotuner's stream-K
        {"name": "fp64_streamk_ragged", "kind": "fp64", "m": 777, "n": 1281, "k": 6001, "odd": True, "call": "gemm",
         "ksplit": 0, "tile_m": 128, "beta": True},
        # SUMMA on a 3 x 5 grid whose blocks differ in size, default panel width
        {"name": "summa_fp64_uneven", "kind": "summa", "m": 3001, "n": 5002, "k": 4096, "rows": 3, "cols": 5,
         "panel": PANEL, "form": "fp64", "splits": 2, "wide": False},
        # digit-slice form at FP64 accuracy, wide exponents
        {"name": "ozaki8_n4096", "kind": "ozaki", "m": 4096, "n": 4096, "k": 4096, "splits": 8, "ksplit": 1,
         "wide": True, "beta": False},
        # the headline product: residue form at FP64 accuracy, N = 16384, wide exponents
        {"name": "crt15_n16384", "kind": "crt", "m": 16384, "n": 16384, "k": 16384, "moduli": 15, "wide": True,
         "beta": False},
        # the same form on an ordinary ragged shape, the middle of the autotuner's range
        {"name": "crt15_ragged", "kind": "crt", "m": 2501, "n": 1999, "k": 3001, "moduli": 15, "wide": True,
         "beta": False},
        # a caller whose matrices are in host memory
        {"name": "host_crt_n4096", "kind": "host", "m": 4096, "n": 4096, "k": 4096, "form": "crt", "splits": 15},
        # the check after every run: all of C against its constant
        {"name": "validate_n8192", "kind": "validate", "m": 8192, "n": 8192},
        # the cost model's training: the autotuner's batch
        {"name": "mlp_step_b256", "kind": "mlp", "batch": 256},
    ]


def _size(rng, lo, hi):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, v // 16 * 16) if rng.random() < 0.5 else v


def _shape(rng, lo, hi, macs):
    """m, n, k in [lo, hi], spread over the logarithm, with m n k at most `macs`."""
    while True:
        m, n, k = (_size(rng, lo, hi) for _ in range(3))
        if m * n * k <= macs:
            return {"m": m, "n": n, "k": k}


def draw(rng):
    kind = rng.choice(["fp64", "fp64", "rows", "chunks", "summa", "ozaki", "crt", "crt", "host", "validate", "mlp"])
    if kind == "fp64":
        c = {"kind": kind, **_shape(rng, 32, 16384, 3e11), "odd": rng.random() < 0.25}
        if rng.random() < 0.5:
            return {**c, "call": "ab"}
        ksplit, tile_m = rng.choice([(1, 128), (1, 64), (2, 128), (4, 128), (8, 64), (0, 128), (0, 128)])
        return {**c, "call": "gemm", "ksplit": ksplit, "tile_m": tile_m, "beta": rng.random() < 0.5}
    if kind == "rows":
        return {"kind": kind, "n": _size(rng, 256, 8000), "ranks": rng.choice([2, 4, 8])}
    if kind == "chunks":
        return {"kind": kind, **_shape(rng, 128, 8192, 2e11), "chunk": rng.choice([256, 512, 1024, CHUNK])}
    if kind == "summa":
        form = rng.choice(["fp64", "fp64", "ozaki", "crt"])
        return {"kind": kind, **_shape(rng, 256, 8192, 1e11), "rows": rng.randint(1, 4), "cols": rng.randint(1, 5),
                "panel": rng.choice([64, 100, PANEL, 512]), "form": form,
                "splits": {"fp64": 2, "ozaki": 8, "crt": 15}[form], "wide": rng.random() < 0.5}
    if kind == "ozaki":
        return {"kind": kind, **_shape(rng, 128, 16384, 3e11), "splits": rng.randint(3, 9),
                "ksplit": rng.choice([1, 1, 4, 16]), "wide": rng.random() < 0.5, "beta": rng.random() < 0.25}
    if kind == "crt":
        return {"kind": kind, **_shape(rng, 128, 16384, 1e12), "moduli": rng.randint(11, 16),
                "wide": rng.random() < 0.5, "beta": rng.random() < 0.25}
    if kind == "host":
        form = rng.choice(["fp64", "ozaki", "crt"])
        return {"kind": kind, **_shape(rng, 256, 6000, 5e10), "form": form,
                "splits": {"fp64": 2, "ozaki": 8, "crt": 15}[form]}
    if kind == "validate":
        return {"kind": kind, "m": _size(rng, 64, 16000), "n": _size(rng, 64, 16000)}
    return {"kind": kind, "batch": _size(rng, 32, 4096)}


# ---------------------------------------------------------------- inputs
def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _matrix(gen, rows, cols, wide=False, odd=False):
    """Uniform [-1, 1), or u 2^e with e a uniform integer in [-20, 20]; `odd`: the row pitch is odd."""
    ld = cols + (1 - cols % 2) if odd else cols
    x = torch.rand((rows, ld), generator=gen, dtype=torch.float64, device="cuda").mul_(2.0).sub_(1.0)
    if wide:
        for r in range(0, rows, 4096):
            e = torch.randint(-20, 21, x[r:r + 4096].shape, generator=gen, device="cuda", dtype=torch.int32)
            x[r:r + 4096] = torch.ldexp(x[r:r + 4096], e)
    return x[:, :cols]


def _cuts(extent, parts):
    """Block boundaries whose sizes differ: part i is about 1 + i / (2 parts) as long as the first."""
    w = [1.0 + 0.5 * i / parts for i in range(parts)]
    c = [0] + [int(round(extent * sum(w[:i + 1]) / sum(w))) for i in range(parts)]
    c[-1] = extent
    return c


def _workspace(nbytes):
    ws = mgx.OzakiWorkspace()
    if nbytes:
        ws.get(nbytes)
    return ws


def _operands(case, seed):
    kind = case["kind"]
    g = _gen(seed, 17)
    m, n = (case["n"], case["n"]) if kind == "rows" else (case["m"], case["n"])
    k = case["n"] if kind == "rows" else case["k"]
    wide = bool(case.get("wide", kind == "host"))
    odd = bool(case.get("odd", False))
    A, B = _matrix(g, m, k, wide, odd), _matrix(g, k, n, wide, odd)
    C = _matrix(g, m, n, wide, odd) if case.get("beta") else None
    return A, B, C


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "validate":
        # a computed C = 2 K with its rounding errors, and a few elements that are wrong
        g = _gen(seed, 5)
        want = 2.0 * case["n"]
        u = torch.rand((case["m"], case["n"]), generator=g, dtype=torch.float64, device="cuda")
        C = want * (1.0 + 4e-16 * u.sub(0.5))
        C += (u > 1.0 - 1e-5) * (want * 1e-9) * u
        return {**s, "C": C, "want": want}
    if kind == "mlp":
        g = _gen(seed, 7)
        b, p = case["batch"], mgx.mlp_param_count()
        X = torch.randn((b, 6), generator=g, device="cuda")
        Y = torch.stack([X[:, 0] + 0.5 * X[:, 1] * X[:, 2], torch.sin(X[:, 5]) - X[:, 3]], dim=1).contiguous()
        P = torch.empty(p, device="cuda").normal_(0.0, 0.15, generator=g)
        # optimiser state of a model in training
        M = torch.empty(p, device="cuda").normal_(0.0, 1e-2, generator=g)
        V = torch.empty(p, device="cuda").uniform_(1e-4, 1e-3, generator=g)
        return {**s, "X": X, "Y": Y, "W": torch.tensor([1.0, 0.5], device="cuda"), "P": P, "M": M, "V": V,
                "G": torch.empty(p, device="cuda"), "L": torch.empty(1, device="cuda"),
                "out": torch.empty((b, 2), device="cuda"), "step": 200}
    A, B, C = _operands(case, seed)
    m, n, k = A.shape[0], B.shape[1], A.shape[1]
    if kind == "host":
        s["A"], s["B"] = A.cpu().pin_memory(), B.cpu().pin_memory()
        s["C"] = torch.empty((m, n), dtype=torch.float64, pin_memory=True)
        return s
    s["A"], s["B"] = A, B
    s["C"] = C if C is not None else torch.empty((m, n), dtype=torch.float64, device="cuda")
    if kind == "fp64" and case["call"] == "gemm":
        ks = case["ksplit"]
        s["ws"] = _workspace(mgx.lib().mgx_fp64_streamk_workspace_size(m, n, k) if ks == 0
                             else mgx.fp64_splitk_workspace_size(m, n, k, ks) if ks > 1 else 0)
    elif kind == "ozaki":
        ks = case["ksplit"]
        s["ws"] = _workspace(mgx.ozaki_splitk_workspace_size(m, n, k, case["splits"], ks) if ks > 1
                             else mgx.ozaki_workspace_size(m, n, k, case["splits"]))
    elif kind == "crt":
        s["ws"] = _workspace(mgx.crt_workspace_size(m, n, k, case["moduli"]))
    elif kind == "summa":
        s["plan"] = mgx.SummaPlan(m, n, k, case["rows"], case["cols"], case["panel"], form=FORMS[case["form"]],
                                  splits=case["splits"], row_cuts=_cuts(m, case["rows"]),
                                  col_cuts=_cuts(n, case["cols"]))
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "validate":
        ok, v = mgx.validate_matrix_c(s["C"], case["m"], case["n"], s["want"])
        return {"passed": bool(ok), "elements": int(v.elements), "invalid": int(v.invalid),
                "max_abs": float(v.max_abs_error), "max_rel": float(v.max_rel_error)}
    if kind == "mlp":
        mgx.mlp_gradients(s["X"], s["Y"], s["W"], s["P"], s["G"], s["L"])
        mgx.mlp_adam_step(s["P"], s["G"], s["M"], s["V"], s["step"], 3e-3)
        mgx.mlp_forward(s["X"], s["P"], s["out"])
        s["step"] += 1
        return {"grads": s["G"], "loss": s["L"], "params": s["P"], "m": s["M"], "v": s["V"], "out": s["out"]}
    A, B, C = s["A"], s["B"], s["C"]
    if kind == "fp64":
        if case["call"] == "ab":
            mgx.ab_multiply(A, B, C)
        else:
            mgx.gemm_fp64(A, B, C, beta_one=case["beta"], ksplit=case["ksplit"], tile_m=case["tile_m"],
                          workspace=s["ws"])
    elif kind == "rows":
        n, ranks = case["n"], case["ranks"]
        cut = [n * r // ranks for r in range(ranks + 1)]
        for r in range(ranks):
            mgx.gemm_fp64(A[cut[r]:cut[r + 1]], B, C[cut[r]:cut[r + 1]])
    elif kind == "chunks":
        m, n, k = case["m"], case["n"], case["k"]
        C.zero_()
        for k0 in range(0, k, case["chunk"]):
            kc = min(case["chunk"], k - k0)
            mgx.ab_multiply_accumulate_async(A, B[k0:k0 + kc], C, m, n, k, k0, kc, k, n, n)
    elif kind == "summa":
        s["plan"].run(A, B, C)
    elif kind == "ozaki":
        mgx.gemm_ozaki(A, B, C, splits=case["splits"], beta_one=case["beta"], workspace=s["ws"],
                       ksplit=case["ksplit"])
    elif kind == "crt":
        mgx.gemm_ozaki_crt(A, B, C, moduli=case["moduli"], beta_one=case["beta"], workspace=s["ws"])
    else:
        mgx.gemm_host(A, B, C, form=FORMS[case["form"]], splits=case["splits"])
        torch.cuda.current_stream().synchronize()   # the caller reads C on the host
    return {"C": C}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "validate":
        e = case["m"] * case["n"]
        return {"bytes": 8.0 * e, "flops": 3.0 * e}
    if kind == "mlp":
        p, b = 4738, case["batch"]
        # forward twice, backward twice a forward; parameters and optimiser state read and written
        return {"bytes": 4.0 * (8 * p + 10 * b), "flops": 2.0 * 4608 * b * 4 + 12.0 * p}
    m, n, k = (case["n"],) * 3 if kind == "rows" else (case["m"], case["n"], case["k"])
    form = case.get("form", kind)
    count = case.get("moduli", case.get("splits", 1))
    products = count * (count + 1) / 2 if form == "ozaki" else count if form == "crt" else 1
    return {"bytes": 8.0 * (m * k + k * n + m * n * (2 if case.get("beta") else 1)),
            "flops": 2.0 * m * n * k * products}


# ---------------------------------------------------------------- the same in plain 64 bits
def _product(A, B):
    """A B in FP64, 1024 columns of A at a time: shorter sums lose less than one long one."""
    C = torch.zeros((A.shape[0], B.shape[1]), dtype=torch.float64, device="cuda")
    for k0 in range(0, A.shape[1], 1024):
        C += A[:, k0:k0 + 1024] @ B[k0:k0 + 1024]
    return C


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed) if kind in ("validate", "mlp") else None
    if kind == "validate":
        err = (s["C"] - s["want"]).abs()
        rel = err / s["want"]
        bad = int(((err > 1e-9) & (rel > 1e-12)).sum())
        return {"passed": bad == 0, "elements": err.numel(), "invalid": bad, "max_abs": float(err.max()),
                "max_rel": float(rel.max())}
    if kind == "mlp":
        X, Y, W = s["X"].double(), s["Y"].double(), s["W"].double()

        def net(p):
            w1, b1, w2, b2, w3, b3 = torch.split(p, [384, 64, 4096, 64, 128, 2])
            h = torch.tanh(X @ w1.view(64, 6).T + b1)
            return torch.tanh(h @ w2.view(64, 64).T + b2) @ w3.view(2, 64).T + b3

        P = s["P"].double().requires_grad_(True)
        loss = ((net(P) - Y).square() * W).sum() / X.shape[0]
        G, = torch.autograd.grad(loss, P)
        M = 0.9 * s["M"].double() + 0.1 * G
        V = 0.999 * s["V"].double() + 0.001 * G * G
        t = s["step"]
        with torch.no_grad():
            P = P - 3e-3 * (M / (1 - 0.9 ** t)) / ((V / (1 - 0.999 ** t)).sqrt() + 1e-8)
            return {"grads": G, "loss": loss.detach().reshape(1), "params": P, "m": M, "v": V, "out": net(P)}
    A, B, C = _operands(case, seed)
    P = _product(A, B)
    if C is not None:
        P += C
    return {"C": P.cpu() if kind == "host" else P}
