"""Forms of a solve that other tests reach no more since most grids take a persistent
sweep, or that none compared with a reference: the tuned line passes, triblocks in 1D and
on tiles, shared launches of unlike grids, the x-tiles at 64 points and past them."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def ps():
    oracle.build()
    import polystring_b200
    return polystring_b200


CHILD = r"""
import json, sys
import numpy as np
sys.path.insert(0, %(root)r)
import polystring_b200 as ps
from polystring_b200 import capi
out = {}
for dim, shape, cell in ((2, (128, 128, 1), ("SQUARE", (8.0,))), (3, (48, 32, 24), ("ORTHORHOMBIC", (4.0, 3.6, 3.2)))):
    rng = np.random.default_rng(5)
    wA = 0.5 * rng.standard_normal(shape)
    wB = -wA + 0.1 * rng.standard_normal(shape)
    m = ps.ModelAB(dim, shape, ps.make_cell(dim, cell[0], *cell[1]), (21, 33), 16.0)
    m.set_fields(wA, wB)
    m.update(2)
    out[str(shape)] = {"H": m.H()[0], "phiA": m.get("phiA").ravel()[::97].tolist(), "n": m.launches_per_propagate()}
out["log"] = capi.load().ps_tuning_log().decode()
print(json.dumps(out))
"""


def _child(tune, sched=None):
    env = dict(os.environ, PS_B200_AUTOTUNE="1" if tune else "0", PS_B200_LINE_PASSES="1")
    if sched is not None:
        env["PS_B200_REG_FFT"] = sched
    r = subprocess.run([sys.executable, "-c", CHILD % {"root": ROOT}], capture_output=True, text=True, env=env,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("sched", [None, "0"])
def test_tuned_line_passes(sched):
    """Another schedule reorders roundings only (two iterations of 52 steps, some 8
    transforms a step, a few eps each: below 1e-12); other tiles change no bit."""
    tuned, plain = _child(True, sched), _child(False, sched)
    assert plain["log"] == ""
    for key in ("(128, 128, 1)", "(48, 32, 24)"):
        a, b = np.array(tuned[key]["phiA"]), np.array(plain[key]["phiA"])
        assert tuned[key]["n"] > 52 and plain[key]["n"] > 52
        assert "grid " + key[1:-1].replace(", ", "x") + " RQM4 batch 1: schedule [" in tuned["log"]
        if sched is None:
            assert abs(tuned[key]["H"] - plain[key]["H"]) <= 1e-12 * abs(plain[key]["H"])
            assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
        else:
            assert tuned[key]["H"] == plain[key]["H"] and np.array_equal(a, b)


@pytest.mark.parametrize("scft", ["EM", "Anderson"])
@pytest.mark.parametrize("dim,shape", [(1, (64, 1, 1)), (1, (24, 1, 1)), (1, (352, 1, 1)), (2, (64, 64, 1)),
                                       (2, (96, 48, 1)), (2, (128, 192, 1)), (2, (12, 352, 1))])
def test_triblocks_match_oracle(ps, dim, shape, scft):
    L = (3.9, 4.3)[:dim]
    w = 0.5 * np.random.default_rng(5).standard_normal((3,) + shape)
    args = (dim, shape)
    rest = ((9, 14, 11), (18.0, 14.0, 25.0))
    o = oracle.ModelABC(*args, L, *rest, scft=scft, n_anderson=3).init_fields(*w)
    m = ps.ModelABC(*args, ps.make_cell(dim, ("LAMELLAR", "RECTANGULAR")[dim - 1], *L), *rest, scft=scft, n_anderson=3)
    m.set_fields(*w)
    o.update(2)
    m.update(2)
    # two iterations of 31 steps, at most 8 line operators each, a few eps of the largest
    # value; the second starts from fields that carry chi = 25 times the first's error
    assert abs(m.Q() - o.Q()) < 1e-11 * o.Q()
    for f in ("phiA", "phiB", "phiC", "wA", "wB", "wC"):
        assert np.abs(m.get(f) - o.get(f)).max() < 1e-11 * max(1.0, np.abs(o.get(f)).max()), f


@pytest.mark.parametrize("long", [False, True])
def test_shared_launches_of_unlike_grids(ps, long):
    """Short axes beside one past 64 points (a CTA an SM) and without it (two)."""
    shapes = [(32, 32, 32), (16, 24, 32), (64, 16, 24), (24, 48, 16), (32, 32, 32), (16, 16, 16)]
    if long:
        shapes += [(96, 16, 24), (16, 24, 128)]
    ortho = lambda s: ps.make_cell(3, "ORTHORHOMBIC", 3.8, 4.0, 4.2)   # noqa: E731
    ab = [dict(dim=3, shape=s, cell=ortho(s), Ms=(9 + 2 * (k % 3), 13), chiN=18.0) for k, s in enumerate(shapes)]
    abc = [dict(dim=3, shape=s, cell=ortho(s), Ms=(9, 8, 9), chi=(18.0, 14.0, 25.0)) for s in shapes[1:3] + shapes[-1:]]
    b = ps.BatchAB(ab, abc)
    assert b.launches_per_propagate() < len(ab) + len(abc)
    rng = np.random.default_rng(2)
    fields = [0.5 * rng.uniform(-1, 1, (3,) + s["shape"]) for s in ab + abc]
    for k, w in enumerate(fields):
        b.set_fields(k, *(w[:2] if k < len(ab) else w))
    b.update(2)
    for k, spec in enumerate(ab + abc):
        m = (ps.ModelAB if k < len(ab) else ps.ModelABC)(**spec)
        m.set_fields(*(fields[k][:2] if k < len(ab) else fields[k]))
        m.update(2)
        assert b.H(k) == m.H()
        for f in ("phiA", "wB"):
            assert np.array_equal(b.get(k, f), m.get(f)), (k, f)


@pytest.mark.parametrize("shape", [(64, 64, 64), (96, 24, 32), (24, 12, 48)])
def test_x_tiles_change_no_bit(ps, monkeypatch, shape):
    w = 0.5 * np.random.default_rng(5).uniform(-1, 1, (2,) + shape)
    out = []
    for v in "012":
        monkeypatch.setenv("PS_B200_SWEEP_VARIANT", v)
        m = ps.ModelAB(3, shape, ps.make_cell(3, "ORTHORHOMBIC", 4.2, 3.9, 4.4), (13, 21), 20.0)
        m.set_fields(*w)
        m.update(2)
        out.append((m.H(), m.get("phiA"), m.get("wB")))
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(o, out[0]))
