"""A stream module's stages in parts: generated from the spec as it is when it is
generated, and for chains of stages of any length."""
import copy

from kunquant_gb300 import codegen
from kunquant_gb300.graph import predefined_spec
from kunquant_gb300.streamgen import tick_groups


def _sources(spec, path):
    return [open(p).read() for p in codegen.generate_module(spec, str(path), tag="parts")]


def test_a_spec_changed_in_place_is_generated_anew(tmp_path):
    spec = predefined_spec("alpha158_stream_f32")
    si = next(i for i, st in enumerate(spec["stages"]) if st["kind"] == "ts" and len(tick_groups(spec)[i][0]) > 1)
    ops = spec["stages"][si]["ops"]
    last = max(i for i, op in enumerate(ops) if op["k"] == "Output")
    assert last == len(ops) - 1
    out = ops.pop()
    short = _sources(spec, tmp_path / "short")
    ops.append(out)
    again = _sources(spec, tmp_path / "again")
    assert again == _sources(copy.deepcopy(spec), tmp_path / "copy") != short


def test_a_long_chain_of_stages():
    n = 3000
    stages = [{"kind": "rank", "in": [k], "out": [k + 1]} for k in range(n)]
    stages.append({"kind": "ts", "in": [n], "out": [n + 1],
                   "ops": [{"k": "Input", "in": [], "buf": n}, {"k": "Abs", "in": [0]},
                           {"k": "Output", "in": [1], "buf": n + 1}]})
    # stages in any order: the last reads what the first ones lead to
    for order in (stages, stages[::-1]):
        si = order.index(stages[-1])
        assert tick_groups({"stages": order}) == {si: [[[1, 2]]]}
