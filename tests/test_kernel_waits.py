"""Bounded waits of the kernels, read from their sources: every one can tell the host that it ran out."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "rpeg_b200" / "csrc"
SOURCES = sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])


def _calls(text, name):
    """Argument lists of the calls of ``name``, split at top-level commas."""
    for m in re.finditer(r"\b%s\(" % name, text):
        depth, args, start = 1, [], m.end()
        for i in range(m.end(), len(text)):
            c = text[i]
            depth += (c in "([{") - (c in ")]}")
            if depth == 0 or (c == "," and depth == 1):
                args.append(text[start:i].strip())
                start = i + 1
            if depth == 0:
                break
        yield args


@pytest.mark.parametrize("source", SOURCES, ids=lambda p: p.name)
def test_waits_have_a_status_word(source):
    places = []
    for args in _calls(source.read_text(), "mbar_wait"):
        if args[0].startswith("uint64_t*"):            # the definition
            continue
        assert len(args) == 5 and args[3].split(".")[-1] == "status", (source.name, args)
        places.append(args[4])
    assert "0" not in places, "a wait names its place"
