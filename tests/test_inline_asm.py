"""Inline PTX of more than one instruction: an output that is written before the block's last read of an
input must be an early clobber ("&"), or the compiler may give both one register."""
import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "hardcaml_zprize_gb300", "csrc", "*.cu*")))


def blocks(text):
    """(template, outputs, inputs) of every asm statement; operands as constraint strings."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"\basm(?:\s+volatile)?\s*\(", text):
        depth, i, in_str, parts, start = 1, m.end(), False, [], m.end()
        while depth:
            ch = text[i]
            if in_str:
                if ch == "\\":
                    i += 1
                elif ch == '"':
                    in_str = False
            elif ch == '"':
                in_str = True
            elif ch == "(":
                depth += 1
            elif ch == ")":
                depth -= 1
            elif ch == ":" and depth == 1:
                if text[i + 1] == ":":  # no outputs
                    parts += [text[start:i], ""]
                    i += 1
                else:
                    parts.append(text[start:i])
                start = i + 1
            i += 1
        parts.append(text[start:i - 1])
        parts += [""] * 3
        template = "".join(re.findall(r'"((?:[^"\\]|\\.)*)"', parts[0])).replace("\\n", "\n").replace("\\t", " ")
        outs = re.findall(r'"([=+][^"]*)"', parts[1])
        ins = re.findall(r'"([a-z])"', parts[2])
        yield template, outs, ins


def unsafe(template, outs, ins):
    """Outputs without "&" that an instruction writes before another one reads an input."""
    insns = [s.strip() for s in re.split(r"[;\n{}]", template) if "%" in s]
    written, last_read = {}, -1
    for k, s in enumerate(insns):
        ops = [int(x) for x in re.findall(r"(?<!%)%(\d+)", s)]
        dest = int(re.match(r"\S+\s+\[?(?<!%)%(\d+)", s).group(1)) if re.match(r"\S+\s+\[?%\d", s) else -1
        if 0 <= dest < len(outs):
            written.setdefault(dest, k)
        if any(len(outs) <= o < len(outs) + len(ins) for o in ops):
            last_read = k
    return [o for o, k in written.items() if k < last_read and "&" not in outs[o]]


def test_the_check_itself():
    assert unsafe("add.u32 %0, %1, 1;\n mul.lo.u32 %0, %0, %1;", ["=r"], ["r"]) == [0]
    assert unsafe("add.u32 %0, %1, 1;\n mul.lo.u32 %0, %0, %1;", ["=&r"], ["r"]) == []
    assert unsafe("add.cc.u32 %0, %2, 1;\n addc.u32 %1, %2, 0;", ["=r", "=r"], ["r"]) == [0]
    assert unsafe("add.u32 %0, %1, %2;", ["=r"], ["r", "r"]) == []


@pytest.mark.parametrize("path", SOURCES, ids=[os.path.basename(p) for p in SOURCES])
def test_early_clobbers(path):
    with open(path) as f:
        text = f.read()
    bad = [(t.split("\n")[0], unsafe(t, o, i)) for t, o, i in blocks(text) if unsafe(t, o, i)]
    assert not bad, bad


def test_blocks_are_found():
    found = 0
    for path in SOURCES:
        with open(path) as f:
            found += sum(1 for _ in blocks(f.read()))
    assert found > 20
