"""Uploads are ordered before the kernels that read them.

Every context works on a stream of its own that does not wait for the legacy
stream, and a copy from pageable memory may return before its data has reached
the device. So no source of the library copies or clears device memory on the
legacy stream, and every kernel is launched on a stream that the launch names.
"""
import os
import re

import pytest

from anns_fhe_b200.build import CSRC, HEADERS, SOURCES

LEGACY = re.compile(r"\bcuda(Memcpy|Memset)(2D|3D|ToSymbol|FromSymbol|ToArray|FromArray|Peer)?\s*\(")


def code(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    text = re.sub(r"/\*.*?\*/", lambda m: "\n" * m.group().count("\n"), text, flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def line_of(text, at):
    return text.count("\n", 0, at) + 1


@pytest.mark.parametrize("name", SOURCES + HEADERS)
def test_no_copy_on_the_legacy_stream(name):
    text = code(name)
    found = [f"{name}:{line_of(text, m.start())}: {m.group()}" for m in LEGACY.finditer(text)]
    assert not found, found


@pytest.mark.parametrize("name", SOURCES + HEADERS)
def test_every_launch_names_its_stream(name):
    text = code(name)
    for m in re.finditer(r"<<<(.*?)>>>", text, flags=re.S):
        depth, parts, part = 0, [], ""
        for ch in m.group(1):
            depth += (ch in "([{") - (ch in ")]}")
            if ch == "," and depth == 0:
                parts.append(part)
                part = ""
            else:
                part += ch
        parts.append(part)
        assert len(parts) == 4, f"{name}:{line_of(text, m.start())}: {m.group()}"
