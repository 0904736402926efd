"""Copies and clears that kernels depend on are ordered before them.

A context's kernels run on its own stream, which does not wait for the default
stream.  A host-to-device copy from pageable memory on the default stream may
still be under way when it returns, and a clear there may not have begun, so a
kernel of the context could read index tables half filled.  That race shows in
few runs; the sources are checked instead: every upload and clear goes to the
context's stream, and blocking copies are made from the device only."""
import pathlib
import re

import pytest

import flowsolversourcecode_b200 as pkg

SOURCES = sorted(p for p in (pathlib.Path(pkg.__file__).parent / "csrc").iterdir() if p.suffix in (".cu", ".cuh"))


def _calls(text, name):
    """Argument texts of the calls of `name` (comments taken out)."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(rf"\b{name}\s*\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_uploads_and_clears_go_to_the_contexts_stream(path):
    text = path.read_text()
    assert not list(_calls(text, "cudaMemset")), "a clear on the default stream"
    assert "cudaStreamLegacy" not in text
    for a in _calls(text, "cudaMemcpy"):
        assert "cudaMemcpyDeviceToHost" in a, f"a copy to the device on the default stream: {a}"
