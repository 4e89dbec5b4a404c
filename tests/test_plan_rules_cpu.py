"""Rules that keep the making of a plan cheap, read from the source (a plan needs a GPU, and
what it copies cannot be seen from outside)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "amdat_gb300", "csrc")


def _body(path, head):
    """the function that starts with `head`, up to its closing brace"""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, path)).read())
    at = text.index(head)
    return text[at:text.index("\n}\n", at)]


def test_slab_rules_on_sizes_come_before_the_members():
    """Plans of few pairs, of small lists and of too many rows are turned away by their
    sizes, before their members (one device copy per unit) are looked at."""
    body = _body("disp.cu", "static void plan_slabs(")
    first = body.index("cudaMemcpy(")
    for rule in ("SLAB_PAIRS", "SLAB_MEAN", "SLAB_ROWS"):
        assert 0 < body.index(rule) < first
    assert "at(N + 1" not in body[:first]
