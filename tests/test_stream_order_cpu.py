"""Work on the default stream that the library's own streams do not wait for:
they are non-blocking, cudaMemset returns before the device has cleared, and a
copy from pageable memory may.  Read from the sources, since a race of this
kind shows on few runs."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "mld-ainv_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cpp"))))
def test_nothing_is_cleared_on_the_default_stream(name):
    assert not re.search(r"\bcudaMemset\(", source(name))


@pytest.mark.parametrize("name,copies", [("layout.cpp", 2), ("hostpipe.cu", 2)])
def test_uploads_have_arrived_when_the_call_returns(name, copies):
    text = source(name)
    at = [m.start() for m in re.finditer(r"\bcudaMemcpy\(", text)]
    assert len(at) == copies
    for a in at:  # the wait comes before the function goes on to use the copy
        assert "cudaStreamSynchronize(nullptr)" in text[a:a + 900], text[a:a + 80]
