"""The table of entry points that the native module calls through (csrc/host/fastops.cpp) against the C functions behind it."""
import re

from zorse_b200.ops import build
from zorse_b200.ops import sm100 as k

KINDS = {"int": "i", "long": "l", "float": "f"}


def _kinds(params, named):
    """A letter per parameter: p for pointers and streams, else of its type; `named`: each ends with a name."""
    out = ""
    for p in (q for q in params.split(",") if q.strip() not in ("", "void")):
        words = [w for w in p.split("=")[0].replace("*", " * ").split() if w != "const"]
        if named and words[-1] != "*":
            words = words[:-1]
        out += "p" if "*" in words or "cudaStream_t" in words else KINDS[" ".join(words)]
    return out


def test_every_member_takes_and_returns_what_its_c_function_does():
    c = {}
    for f in build.sources():
        text = re.sub(r"//[^\n]*", "", f.read_text())
        for m in re.finditer(r"\b(int|void|const char\s*\*)\s*(zb_\w+)\s*\(([^)]*)\)\s*\{", text):
            assert m.group(2) not in c, m.group(2)
            c[m.group(2)] = m.group(1).replace(" ", ""), m.group(3)
    src = build.FAST_SRC.read_text()
    body = re.sub(r"//[^\n]*", "", src[src.index("struct Entry {"):src.index("Entry lib;")])
    members = re.findall(r"(int|void|const char\s*\*)\s*\(\*(\w+)\)\(([^)]*)\);", body)
    assert len(members) == len(k._FAST_ENTRIES)
    for name, (returns, member, params) in zip(k._FAST_ENTRIES, members):
        assert name in c, name
        assert (returns.replace(" ", ""), _kinds(params, False)) == (c[name][0], _kinds(c[name][1], True)), name
