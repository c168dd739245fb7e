"""Scale at the edges of its 64-value steps, against the oracle's sequential sum."""
import numpy as np
import pytest

from kunquant_gb300 import build, runner as kr
from oracle.oracle import OracleProgram
from tests import golden_util as G
from tests.parity import compare_exact


def _scale_spec(dtype):
    spec = {"name": "scale_unit_" + dtype, "dtype": dtype, "input_layout": "TS", "output_layout": "TS",
            "blocking_len": 8, "aligned": False, "options": {},
            "buffers": [{"id": 0, "name": "a", "kind": "INPUT", "num_users": 1, "unreliable_count": 0, "window": 1},
                        {"id": 1, "name": "out", "kind": "OUTPUT", "num_users": 0, "unreliable_count": 0,
                         "window": 1}],
            "stages": [{"name": "scale", "kind": "scale", "in": [0], "out": [1], "deps": [], "pending": 0,
                        "ops": [{"k": "Input", "in": [], "buf": 0, "p": -1}, {"k": "Scale", "in": [0], "p": -1},
                                {"k": "Output", "in": [1], "buf": 1, "p": -1}]}]}
    return spec


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float", "double"])
@pytest.mark.parametrize("S", [1, 31, 32, 33, 63, 64, 65, 127, 129, 2049, 8191, 12000])
def test_scale_rows(dtype, S):
    spec = _scale_spec(dtype)
    lib = kr.Library.load(build.build_module_library([spec], "kun_" + spec["name"]))
    rng = np.random.default_rng(S)
    a = rng.standard_normal((4, S)).astype(np.float32 if dtype == "float" else np.float64)
    a[1, rng.random(S) < 0.3] = np.nan
    a[2] = 0.0
    a[3, ::2] *= 1e6
    got = kr.runGraph(kr.createSingleThreadExecutor(), lib.getModule(spec["name"]), {"a": a}, 0, 4)
    assert not compare_exact(got, OracleProgram(spec).run({"a": a}))
