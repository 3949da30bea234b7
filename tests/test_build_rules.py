"""The Makefile's rules name every header that the sources include, so that a change of one rebuilds them."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bbarolo2_gb300", "csrc")


def _includes(name, seen):
    for h in re.findall(r'^#include "([^"]+)"', open(os.path.join(CSRC, name)).read(), re.M):
        if h not in seen:
            seen.add(h)
            if os.sep not in h and "/" not in h:
                _includes(h, seen)
    return seen


def test_every_header_is_a_prerequisite():
    rules = dict(re.findall(r"^\$\(OBJDIR\)/%\.o: %(\.\w+) (.*)$", open(os.path.join(CSRC, "Makefile")).read(), re.M))
    files = [f for f in os.listdir(CSRC) if os.path.splitext(f)[1] in rules]
    assert files and set(rules) == {".cu", ".cpp"}
    for f in files:
        named = set(rules[os.path.splitext(f)[1]].split())
        assert _includes(f, set()) - {os.path.basename(n) for n in named} - named == set(), f
