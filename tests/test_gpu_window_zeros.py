"""Order statistics of windows that hold zeros of both signs: equal in every
comparison, the one that stands at the place asked for is returned as it was
put in.  Float and double, against the oracle bit for bit."""
import numpy as np
import pytest

from kunquant_gb300 import build, runner as kr
from oracle.oracle import OracleProgram
from tests.parity import compare_exact


def _spec(dtype, W):
    ops = [{"k": "Input", "in": [], "buf": 0}, {"k": "BackRef", "in": [0], "window": W},
           {"k": "SkipListState", "in": [1, 0], "window": W},
           {"k": "SkipListMin", "in": [2]}, {"k": "SkipListMax", "in": [2]}, {"k": "SkipListArgMin", "in": [2]},
           {"k": "SkipListRank", "in": [2, 0]}, {"k": "SkipListQuantile", "in": [2], "q": "0.5"},
           {"k": "SkipListQuantile", "in": [2], "q": "0.37"}]
    names = ["min", "max", "argmin", "rank", "q50", "q37"]
    ops = [dict({"p": -1}, **o) for o in ops]
    ops += [{"k": "Output", "in": [3 + k], "p": -1, "buf": k + 1} for k in range(len(names))]
    bufs = [{"id": 0, "name": "a", "kind": "INPUT", "num_users": 1, "unreliable_count": 0, "window": W + 1}]
    bufs += [{"id": k + 1, "name": n, "kind": "OUTPUT", "num_users": 0, "unreliable_count": 0, "window": 1}
             for k, n in enumerate(names)]
    name = f"window_zeros_{dtype}_{W}"
    return {"name": name, "dtype": dtype, "input_layout": "TS", "output_layout": "TS", "blocking_len": 8,
            "aligned": False, "options": {}, "buffers": bufs, "single_value_inputs": [],
            "stages": [{"name": name, "kind": "ts", "in": [0], "out": [b["id"] for b in bufs[1:]], "deps": [],
                        "pending": 0, "ops": ops}]}


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float", "double"])
@pytest.mark.parametrize("W", [3, 11])
def test_zeros_of_both_signs(dtype, W):
    spec = _spec(dtype, W)
    lib = kr.Library.load(build.build_module_library([spec], "kun_" + spec["name"]))
    rng = np.random.default_rng(W)
    T, S = 150, 64
    zero = np.where(rng.random((T, S)) < 0.5, -0.0, 0.0)
    a = np.where(rng.random((T, S)) < np.linspace(0, 1, S), zero, np.floor(3 * rng.standard_normal((T, S))))
    a[rng.random((T, S)) < 0.01] = np.nan
    a[:, 5::9] = np.where(rng.random(a[:, 5::9].shape) < 0.1, 5e-324 if dtype == "double" else 1e-45, a[:, 5::9])
    a[:, 7::9] = np.where(rng.random(a[:, 7::9].shape) < 0.1, -np.inf, a[:, 7::9])
    a = a.astype(np.float32 if dtype == "float" else np.float64)
    got = kr.runGraph(kr.createSingleThreadExecutor(), lib.getModule(spec["name"]), {"a": a}, 0, T)
    bad = compare_exact(got, OracleProgram(spec).run({"a": a}))
    assert not bad, bad
