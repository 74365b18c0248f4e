"""Rules of the inline PTX, checked on the source text (no GPU needed): the compiler may move an asm
statement that is not volatile, and one between the instructions of a carry chain would change the
flag; and it may give an input the register of an output that is not marked early-clobbered."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cusnarks_b200", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
STRING = re.compile(r'"((?:[^"\\]|\\.)*)"')


def _statements(path):
    """(line, volatile, instructions, constraints of the outputs) of each asm statement."""
    text = open(path).read().replace("\\\n", "  ")
    for m in re.finditer(r"\basm\b\s*(volatile)?\s*\(", text):
        depth, i, quoted = 1, m.end(), False
        while depth:
            c = text[i]
            if c == '"' and text[i - 1] != "\\":
                quoted = not quoted
            elif not quoted:
                depth += (c == "(") - (c == ")")
            i += 1
        body = text[m.end():i - 1]
        template, rest = "", body.lstrip()
        while rest.startswith('"'):
            s = STRING.match(rest)
            template += s.group(1)
            rest = rest[s.end():].lstrip()
        template = template.replace("\\n", " ").replace("\\t", " ").strip("{} ")
        ins = [x.strip() for x in template.split(";") if x.strip(" {}")]
        outs = rest[1:].split(":")[0] if rest.startswith(":") else ""
        yield text.count("\n", 0, m.start()) + 1, bool(m.group(1)), ins, STRING.findall(outs)


@pytest.mark.parametrize("name", FILES)
def test_statements_that_touch_the_carry_flag_are_volatile(name):
    for line, volatile, ins, _ in _statements(os.path.join(CSRC, name)):
        ops = [x.split()[0].split(".") for x in ins]
        flag = any("cc" in op or op[0] in ("addc", "subc", "madc") for op in ops)
        assert volatile or not flag, f"{name}:{line}"


@pytest.mark.parametrize("name", FILES)
def test_outputs_written_before_the_last_input_are_early_clobbered(name):
    for line, _, ins, outs in _statements(os.path.join(CSRC, name)):
        args = [[int(k) for k in re.findall(r"%(\d+)", x)] for x in ins]
        last_input = max([i for i, a in enumerate(args) if any(k >= len(outs) for k in a)], default=-1)
        for k, constraint in enumerate(outs):
            written = min(i for i, a in enumerate(args) if a and a[0] == k)
            assert written >= last_input or "&" in constraint, f"{name}:{line}: operand {k}"


def test_local_points_read_16_bytes_at_a_time_are_aligned():
    """lds_fq reads uint4: an array on the stack that goes to it, or to the out-of-line addition that
    calls it, has no such alignment of itself."""
    text = open(os.path.join(CSRC, "group.cuh")).read()
    arrays = re.findall(r"^(.*)\buint32_t (\w+)\[[^\]]+\];", text, re.M)
    assert arrays
    for before, name in arrays:
        if "__align__(16)" not in before:
            assert not re.search(r"\b(?:lds_fq|group_add_slow<F>)\([^;]*\b%s\b" % name, text), name


def test_statements_are_found():
    n = sum(len(list(_statements(os.path.join(CSRC, f)))) for f in FILES)
    assert n >= 10
