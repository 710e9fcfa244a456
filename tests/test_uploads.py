"""Uploads outlive their sources: an asynchronous host-to-device copy may still read its source after the call
returned (always from pinned memory, and from pageable memory that the GPU can read itself), so the source must be
pinned staging that is kept, or the function must wait before it returns."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "omnioperator_gb300" / "csrc"

# Sources that live on in the caller or the factory: who waits for the copy.
KEPT = {
    ("sizer.cpp", "X"): "Predict and Train read results back before they return",
    ("sizer.cpp", "T"): "Train reads the loss back before it returns",
    ("hash_join.cpp", "f_.filterText.data()"): "a member of the factory, which outlives its operators",
}


def _functions(text):
    """(start, end) of top-level function bodies: from a line that is `{` to the next that is `}`."""
    opens = [m.start() for m in re.finditer(r"^\{$", text, re.M)]
    return [(o, text.index("\n}", o)) for o in opens]


def _uploads():
    for path in sorted(CSRC.rglob("*.c*")):
        text = path.read_text()
        for m in re.finditer(r"cudaMemcpyAsync\(([^;]*?),\s*cudaMemcpyHostToDevice", text, re.S):
            args = re.split(r",\s*(?![^()]*\))", m.group(1))
            yield path.name, text, m, args[1].strip()


def _pinned(body, source):
    name = re.match(r"([\w.\->]+?)(?:\.Get\(\))$", source)
    if not name:
        return False
    last = re.split(r"\.|->", name.group(1))[-1]
    return any(re.search(r"PinnedArray<[^;]*>[^;()]*\b%s\b" % re.escape(last), f.read_text())
               for f in CSRC.rglob("*") if f.suffix in (".h", ".cpp"))


@pytest.mark.parametrize("site", list(_uploads()), ids=lambda s: f"{s[0]}-{s[3]}")
def test_source_outlives_the_copy(site):
    name, text, m, source = site
    start, end = next((f for f in _functions(text) if f[0] <= m.start() < f[1]), (0, len(text)))
    body, rest = text[start:end], text[m.end():end]
    static = re.search(r"static const[^;]*\b%s\b" % re.escape(source), body)
    waits = re.search(r"\bSync\(\)|cudaStreamSynchronize", rest)
    assert static or waits or _pinned(body, source) or (name, source) in KEPT, f"{name}: {source}"


def test_every_upload_is_looked_at():
    total = sum(p.read_text().count("cudaMemcpyHostToDevice") for p in CSRC.rglob("*.c*"))
    assert total == len(list(_uploads())) > 10
