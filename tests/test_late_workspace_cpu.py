"""finish (csrc/host/fastops.cpp) asks the allocator for nothing once its first product is launched: a product that starts under
others may not write to memory that was given back while they were queued."""
import re

from zorse_b200.ops import build


def test_the_workspaces_of_a_list_are_taken_ahead_of_its_first_launch():
    src = build.FAST_SRC.read_text()
    body = src[src.index("PyObject* finish("):]
    body = body[:re.search(r"\n}\n", body).end()]
    first = min(body.index(" gemm("), body.index("launch("))
    assert "split_workspace(" in body[:first] and not re.search(r"split_workspace\(|\bempty\(", body[first:])
    call = re.search(r"\bgemm\(([^;]*)\);", body).group(1)
    assert call.endswith("&workspaces[launched]")               # (nullptr would have gemm ask for one of its own)
