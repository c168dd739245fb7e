"""Rank on rows at the edges of its block sizes, over value distributions that
take each of its ways: spread values, ties alone and among other values,
infinities, values that need the other bucket map, a refined map or the sort.
The result is an integer count divided twice, so it is compared bit for bit."""
import numpy as np
import pytest

from kunquant_gb300 import build, runner as kr
from oracle.oracle import OracleProgram
from tests import golden_util as G
from tests.parity import compare_exact

_mods = {}


def _module(fixture):
    if fixture not in _mods:
        spec = G.load(fixture)[0]
        lib = kr.Library.load(build.build_module_library([spec], "kun_rank_" + fixture))
        _mods[fixture] = (lib, lib.getModule(spec["name"]), spec)
    return _mods[fixture][1:]


def _rows(S, rng):
    n = rng.normal(size=S)
    i = np.arange(S)
    rows = [n, np.exp(13 + n), rng.random(S), np.floor(rng.random(S) * 10) / 10, np.full(S, 3.5),
            np.tan(3.14 * (rng.random(S) - 0.5)),
            np.where(i == S // 2, 1e30, n),                                    # one far value
            np.where(i % 50 == 0, np.where(i % 100 == 0, -np.inf, np.inf), n),
            np.where(i % 2 == 0, np.inf, -np.inf),
            1e-40 * np.floor(rng.random(S) * 1000),                            # denormals
            np.where(i % 2 == 0, 1e-8 * n, 1e8 * (1 + 1e-7 * n)),              # two tight clusters
            np.where(rng.random(S) < 0.5, -1, 1) * np.exp(20 * n),             # both signs, many binades
            np.where(i % 10 < 3, -0.0, np.where(i % 10 < 5, 0.0, n)),          # ties among spread values
            np.exp(3 * n), np.full(S, np.nan)]
    # many ties at one value inside a cluster that one bucket holds, beside a wide range
    rows.append(np.where(i % 64 == 0, 1e6 * rng.random(S), np.where(i % 3 == 0, 1.0, 1 + 1e-6 * i)))
    out = np.stack(rows)
    out[:, 1::97] = np.where(rng.random(out[:, 1::97].shape) < 0.5, np.nan, out[:, 1::97])
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("fixture", ["rank_ties_nan", "rank029_f64"])
@pytest.mark.parametrize("S", [1, 2, 31, 33, 127, 128, 129, 256, 257, 997, 1025, 4096, 4097, 5001, 8192, 8193, 16384])
def test_rank_rows(fixture, S):
    mod, spec = _module(fixture)
    dt = np.float32 if spec["dtype"] == "float" else np.float64
    with np.errstate(over="ignore"):
        a = _rows(S, np.random.default_rng(S)).astype(dt)
    got = kr.runGraph(kr.createSingleThreadExecutor(), mod, {"a": a}, 0, len(a))
    bad = compare_exact(got, OracleProgram(spec).run({"a": a}))
    assert not bad, dict(list(bad.items())[:5])
