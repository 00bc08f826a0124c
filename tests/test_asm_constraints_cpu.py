"""Inline assembly of several instructions: an output that is written while an
input is still to be read must be an early clobber ("=&r", "+&r"), or the
compiler may give both one register.  Read from the sources; no GPU."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gpupi_b200" / "csrc"
SOURCES = sorted(p.name for p in CSRC.glob("*.cu*"))


def statements(text):
    """(line, template, outputs, inputs) of every asm statement."""
    for m in re.finditer(r"\basm\s*(?:volatile)?\s*\(", text):
        depth, i, quoted = 1, m.end(), False
        parts = [""]
        while depth:
            c = text[i]
            if c == '"' and text[i - 1] != "\\":
                quoted = not quoted
            if not quoted:
                depth += (c == "(") - (c == ")")
                if c == ":" and depth == 1:
                    if text[i - 1] != ":" and text[i + 1] != ":":
                        parts.append("")
                        i += 1
                        continue
                    if text[i + 1] == ":" and text[i + 2] != ":" and parts[-1].rstrip().endswith('"'):
                        parts += ["", ""]   # "::": no outputs
                        i += 2
                        continue
            if depth:
                parts[-1] += c
            i += 1
        constraints = [re.findall(r'"([^"]*)"\s*\(', p) for p in parts[1:3]] + [[], []]
        template = "".join(re.findall(r'"((?:[^"\\]|\\.)*)"', parts[0]))
        yield text.count("\n", 0, m.start()) + 1, template, constraints[0], constraints[1]


def missing_clobbers(text):
    out = []
    for line, template, outputs, inputs in statements(text):
        code = [s for s in re.sub(r"\\[nt]", " ", template).split(";") if s.strip()]
        ops = [[int(n) for n in re.findall(r"%(\d+)", s)] for s in code]
        for k, c in enumerate(outputs):
            writes = [i for i, o in enumerate(ops) if o and o[0] == k]
            if not writes or "&" in c:
                continue
            later = [o for i in range(writes[0] + 1, len(ops)) for o in ops[i]]
            if any(n in later for n in range(len(outputs), len(outputs) + len(inputs))):
                out.append((line, k, c))
    return out


def test_reader():
    text = '''asm("add.cc.u32 %0, %2, %3;\\n\\taddc.u32 %1, %4, 0;" : "=r"(a), "=r"(b) : "r"(x), "r"(y[f(1)]), "r"(z));
              asm volatile("bar.sync %0, 256;" ::"r"(id) : "memory");'''
    (l0, t0, o0, i0), (l1, t1, o1, i1) = statements(text)
    assert (l0, o0, i0) == (1, ["=r", "=r"], ["r"] * 3) and (l1, o1, i1) == (2, [], ["r"])
    assert missing_clobbers(text) == [(1, 0, "=r")]
    assert missing_clobbers(text.replace('"=r"(a)', '"=&r"(a)')) == []


@pytest.mark.parametrize("name", SOURCES)
def test_early_clobbers(name):
    assert missing_clobbers((CSRC / name).read_text()) == []
