"""The persistent delta kernel rewrites the lists that it has counted, within one launch. So its reads of them
must not take the read-only load path, which holds only for data that no thread writes meanwhile."""
import os
import re

SRC = os.path.join(os.path.dirname(__file__), "..", "custingeralg_b200", "csrc", "tc_stream.cu")


def _body(text, name):
    at = re.search(r"\b%s\([^;{]*\)\s*\{" % name, text)
    assert at, name
    return text[at.end():text.index("\n}\n", at.end())]


def test_lists_that_the_launch_rewrites_are_read_by_plain_loads():
    text = open(SRC).read()
    read_only = ("__ldg", "ld.global.nc", "lower_bound(L")
    parts = {n: _body(text, n) for n in ("warp_lower_bound", "delta_part", "delta_count", "compact_vertex",
                                         "grid_meet", "k_delta_fused")}
    # the merge walks start with a read-only search; only the launches that rewrite nothing compile them
    parts["delta_range"], merge = _body(text, "delta_range").split("else if (PRED == kPredBatch) {")
    assert "lower_bound(L" in merge
    for name, body in parts.items():
        for way in read_only:
            plain = body.replace("warp_lower_bound(L", "")
            assert way not in plain, (name, way)
