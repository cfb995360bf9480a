"""Inline PTX that touches memory says so to the compiler: without a "memory" clobber an access may be moved
across the stores, barriers and waits around it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "complab3d-gems_b200", "csrc")
TOUCHES_MEMORY = re.compile(r"\b(ld|st|cp|red|atom|mbarrier|fence|membar|griddepcontrol)\.")


def statements(text):
    """The asm statements of a source, each as its text up to the closing parenthesis."""
    for m in re.finditer(r"\basm\s*(volatile)?\s*\(", text):
        depth, i, quoted = 1, m.end(), False
        while depth:
            c = text[i]
            if c == '"' and text[i - 1] != "\\":
                quoted = not quoted
            elif not quoted:
                depth += (c == "(") - (c == ")")
            i += 1
        yield text[m.start():i]


def test_memory_accesses_in_asm_are_ordered():
    found, bad = 0, []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        for s in statements(open(path).read()):
            if TOUCHES_MEMORY.search(s):
                found += 1
                if "volatile" not in s or '"memory"' not in s:
                    bad.append((os.path.basename(path), s.split("\n")[0]))
    assert found > 10 and not bad, bad
