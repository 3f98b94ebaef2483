"""Programmatic dependent launch guard for kernels picked by a function
(static, CPU).

solver.cu launches the transforms and the stretched grids' line solve through
functions that return the kernel of a length (``launch_k(s->pdl,
dft_fwd_kernel(L), ...)``).  These kernels too must wait for their predecessor
before touching memory: the first statement of each is pdl_enter(), or the
griddepcontrol.wait it stands for, in whichever source file it is defined.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "simplevofsolver_b200", "csrc")
TEXTS = {os.path.basename(p): open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu*"))}
WAITS = re.compile(r'(pdl_enter\(\)|asm volatile\("griddepcontrol\.wait;" ::: "memory"\))$')


def closing(text, start):
    """the index of the bracket that closes the one at `start`"""
    pairs, depth = {"(": ")", "{": "}"}, 0
    for i in range(start, len(text)):
        depth += {text[start]: 1, pairs[text[start]]: -1}.get(text[i], 0)
        if 0 == depth:
            return i
    raise AssertionError("unbalanced brackets")


def launched(texts):
    """the kernels of every launch_k(s->pdl, ...), those of a selector by the
    addresses that its definition takes"""
    names = set()
    for launch in re.findall(r"launch_k\(\s*s->pdl\s*,\s*([^,]+),", texts["solver.cu"]):
        m = re.match(r"(\w+)\s*(\()?", launch)
        if not m.group(2):
            names.add(m.group(1))
            continue
        found = set()
        for text in texts.values():
            for d in re.finditer(r"\w+ " + m.group(1) + r"\(", text):
                end = closing(text, d.end() - 1)
                if text[end + 1:].lstrip().startswith("{"):
                    body = text[text.index("{", end):]
                    found |= set(re.findall(r"&(?:\w+::)*(k\w*_\w+)", body[:closing(body, 0)]))
        assert found, launch
        names |= found
    return names


def first_statement(kernel, texts):
    for text in texts.values():
        for m in re.finditer(r"__global__\s+void[^;{]*?\b" + kernel + r"\s*\(", text):
            end = closing(text, m.end() - 1)
            if text[end + 1:].lstrip().startswith("{"):
                body = re.sub(r"//[^\n]*", "", text[text.index("{", end) + 1:])
                return body.strip().split(";\n", 1)[0].strip()
    raise AssertionError(f"definition of {kernel} not found")


def unguarded(texts):
    return {k for k in launched(texts) if not WAITS.match(first_statement(k, texts))}


SELECTED = ("k_dct_fwd", "k_dct_inv", "k_dft_fwd", "k_dft_inv", "k_cline_solve")


def test_selected_kernels_are_seen():
    assert set(SELECTED) | {"k_geom", "k_predict", "k_project"} <= launched(TEXTS)


def test_every_launched_kernel_waits_first():
    assert not unguarded(TEXTS)


@pytest.mark.parametrize("kernel", SELECTED)
def test_a_missing_wait_is_found(kernel):
    # the sources with that kernel's wait taken out, as text
    texts = dict(TEXTS)
    for name, text in TEXTS.items():
        m = re.search(r"__global__\s+void[^;{]*?\b" + kernel + r"\s*\([^;{]*\)\s*\{", text)
        if m:
            cut = re.search(r"(pdl_enter\(\)|asm volatile\(\"griddepcontrol[^;]*;[^;]*\));\n", text[m.end():])
            texts[name] = text[:m.end()] + text[m.end():].replace(cut.group(0), "", 1)
            break
    assert unguarded(texts) == {kernel}
