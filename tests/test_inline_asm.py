"""Inline PTX statements of more than one instruction: an output that an earlier
instruction writes while a later one still reads an input must be declared early
clobber ("=&r"), or the compiler may give both the same register."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "tensorkyber_b200", "csrc")
SOURCES = sorted(p for ext in ("cu", "cuh", "h", "cpp") for p in glob.glob(f"{CSRC}/*.{ext}"))


def statements(text):
    """(template, outputs, inputs) of every asm statement: constraint lists."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"\basm\s*(?:volatile\s*)?\(", text):
        parts, depth, i, cur = [], 1, m.end(), ""
        while depth:
            c = text[i]
            if c == '"':
                j = i + 1
                while text[j] != '"':
                    j += 2 if text[j] == "\\" else 1
                cur += text[i:j + 1]
                i = j + 1
                continue
            depth += (c in "([") - (c in ")]")
            if c == ":" and depth == 1:
                parts.append(cur)
                cur = ""
            elif depth:
                cur += c
            i += 1
        parts.append(cur)
        strings = [re.findall(r'"((?:[^"\\]|\\.)*)"', p) for p in parts]
        yield ("".join(strings[0]), strings[1] if len(strings) > 1 else [],
               strings[2] if len(strings) > 2 else [])


def hazards(template, outputs, inputs):
    """Outputs written before the last read of some input, without early clobber."""
    uses = [[int(n) for n in re.findall(r"(?<!%)%(\d+)", ins)]
            for ins in template.replace("\\n", " ").replace("\\t", " ").split(";")]
    last_read = max([i for i, u in enumerate(uses) if any(n >= len(outputs) for n in u)],
                    default=-1)
    return [o for o, c in enumerate(outputs) if "&" not in c
            and next(i for i, u in enumerate(uses) if o in u) < last_read]


def test_the_check_itself():
    two = "ld.u32 %0, [%2];\\n\\tld.u32 %1, [%3];"
    assert hazards(two, ["=r", "=r"], ["r", "r"]) == [0]
    assert hazards(two, ["=&r", "=r"], ["r", "r"]) == []
    got = list(statements('asm volatile("a %0, [%1];"\n "b;" : "=r"(x[1]) : "r"(f(y)) : "memory");'))
    assert got == [("a %0, [%1];b;", ["=r"], ["r"])]


@pytest.mark.parametrize("path", SOURCES, ids=[os.path.basename(p) for p in SOURCES])
def test_outputs_written_before_inputs_are_read_are_early_clobber(path):
    with open(path) as f:
        for template, outputs, inputs in statements(f.read()):
            assert hazards(template, outputs, inputs) == [], template
