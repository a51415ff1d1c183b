"""Warp collectives in inline PTX are `asm volatile`.

A collective has to be executed where every lane of its mask is.  The compiler
may move an `asm` without `volatile` to where its result is used (or drop it);
under a branch on the lane that would leave one lane waiting for the others.
Checked on the sources: no device.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "self-join-hpbdc2019_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
# what all lanes of a warp (or threads of a block) have to reach together
COLLECTIVE = re.compile(r"\.sync\b|\.aligned\b|\bbar\.|\bbarrier\.")


def _asm_statements(text):
    text = re.sub(r"//[^\n]*", " ", text)
    return re.findall(r"\basm\s*(volatile|__volatile__)?\s*\(\s*((?:\"(?:[^\"\\]|\\.)*\"\s*)+)", text)


@pytest.mark.parametrize("name", SOURCES)
def test_collectives_are_volatile(name):
    for volatile, code in _asm_statements(open(os.path.join(CSRC, name)).read()):
        assert volatile or not COLLECTIVE.search(code), f"{name}: asm without volatile: {code.strip()}"


def test_the_statements_are_found():
    found = [code for name in SOURCES for _, code in _asm_statements(open(os.path.join(CSRC, name)).read())]
    assert any("redux.sync" in code for code in found) and len(found) > 5
