"""On several streams the order of a module's kernels comes from the module's
table alone: per kernel the series it reads from others and those it writes.  A
read that the table misses would be a race without an error.  This holds the
tables of the shipped batch modules against the pointers that the generated
kernels load from and store to."""
import re

import pytest

from kunquant_gb300 import codegen
from kunquant_gb300.graph import predefined_spec

KEYS = ["alpha101_f32", "alpha158_f32", "alpha158_f64", "alpha158_slide_f32", "alpha158_plain_f32",
        "alpha101_fast_f32", "alpha158_fast_f32"]
POINTER = re.compile(r"\bb(\d+) = \((?:const )?\w+\*\)P\.([pw])\[(\d+)\]")


def _table(numbers, kernels):
    """[(reads, writes)] of a stage's kernel_info array."""
    q, out = kernels, []
    for _ in range(kernels):
        q += 1  # instructions
        lists = []
        for _ in range(2):
            n = numbers[q]
            lists.append(set(numbers[q + 1:q + 1 + n]))
            q += 1 + n
        out.append(tuple(lists))
    assert q == len(numbers)
    return out


def _functions(src, prefix):
    """{kernel index: text of its body and of its staged instance}"""
    out = {}
    heads = [(m.start(), m.group(2), m.group(3)) for m in re.finditer(
        r"(void (?:__launch_bounds__\([^)]*\) )?)(%s_L\d+_\d+)(\w*)\(" % re.escape(prefix), src)
        if m.group(3) in ("_body", "_tma")]
    for start, name, kind in heads:
        end = src.index("\n}\n", start)
        out.setdefault(int(name.rsplit("_", 1)[1]), []).append((kind, src[start:end]))
    return out


def _touched(kind, text):
    """Series a kernel loads from and stores to, as ("p" or "w", slot)."""
    reads, writes = set(), set()
    where = {}
    for j, space, slot in POINTER.findall(text):
        assert where.setdefault(j, (space, int(slot))) == (space, int(slot)), "one pointer name for two series"
    body = POINTER.sub("", text)
    for m in re.finditer(r"\bb(\d+)\b(\[)?", body):
        if m.group(1) not in where:
            continue
        end = m.end()
        if m.group(2):
            depth = 1
            while depth:
                depth += {"[": 1, "]": -1}.get(body[end], 0)
                end += 1
        store = m.group(2) and re.match(r" = ", body[end:])
        (writes if store else reads).add(where[m.group(1)])
    # pointers used without a name (bulk copies)
    for space, slot in re.findall(r"P\.([pw])\[(\d+)\]", body):
        reads.add((space, int(slot)))
    return reads, writes


@pytest.mark.parametrize("key", KEYS)
def test_table_has_what_the_kernels_touch(key, tmp_path):
    spec = predefined_spec(key)
    tag = spec["name"]
    src = "\n".join(open(p).read() for p in codegen.generate_module(spec, str(tmp_path), tag=tag))
    inputs = {b["id"] for b in spec["buffers"] if b["kind"] == "INPUT"}
    checked = 0
    for m in re.finditer(r"st(\d+)_kinfo\[\] = \{([^}]*)\}", src):
        prefix = f"kst_{tag}_{m.group(1)}"
        kernels = _functions(src, prefix)
        table = _table([int(v) for v in m.group(2).split(",")], len(kernels))
        launch = src[src.index(f'int {prefix}_launch('):]
        buffer = {int(s): int(b) for s, b in re.findall(r"P\.p\[(\d+)\] = a->buffers\[(\d+)\];",
                                                        launch[:launch.index("\n}\n")])}

        def series(places):
            return {buffer[slot] if space == "p" else -1 - slot for space, slot in places}

        for k, bodies in kernels.items():
            for kind, text in bodies:
                reads, writes = (series(x) for x in _touched(kind, text))
                if kind == "_tma":
                    reads -= table[k][1]  # the addresses of its outputs too
                else:
                    assert writes == table[k][1], (prefix, k)
                assert reads - inputs - writes <= table[k][0], (prefix, k, kind)
                assert writes <= table[k][1], (prefix, k, kind)
                checked += 1
    assert checked > 50, checked


@pytest.mark.parametrize("key", ["alpha158_f32", "alpha158_slide_f32", "alpha101_f32"])
def test_table_says_which_kernels_have_a_capped_instance(key, tmp_path):
    spec = predefined_spec(key)
    tag = spec["name"]
    src = "\n".join(open(p).read() for p in codegen.generate_module(spec, str(tmp_path), tag=tag))
    seen = set()
    for m in re.finditer(r"st(\d+)_kinfo\[\] = \{([^}]*)\}", src):
        prefix = f"kst_{tag}_{m.group(1)}"
        info = [int(v) for v in m.group(2).split(",")]
        for k in _functions(src, prefix):
            capped = re.search(r"%s_L\d+_%d_r\(" % (re.escape(prefix), k), src) is not None
            assert bool(info[k] & 0x40000000) == capped, (prefix, k)
            seen.add(capped)
    assert seen == {False, True}


def test_the_check_sees_a_missing_read(tmp_path):
    text = "  const float* __restrict__ b3 = (const float*)P.p[2] + s;\n  float* __restrict__ b4 = (float*)P.w[7] + s;\n" \
           "  b4[(t + u) * st4] = kun::ldw<KE>(b3, st3, (long long)(t + u), length) + b4[(t - 1) * st4];"
    assert _touched("_body", text) == ({("p", 2), ("w", 7)}, {("w", 7)})
