"""Host-to-device copies of the library are ordered before the kernels that read them.

The kernels run on non-blocking streams, which do not wait for the legacy stream; a plain
cudaMemcpy from pageable memory runs there and may return before its transfer has landed.
So every such copy goes on the context's stream, or the legacy stream is waited for.  A
missing order shows on no particular run, so this reads the source."""

import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tonto_b200", "csrc")


def _code(name):
    txt = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", txt)


@pytest.mark.parametrize("name", ["tontofock.cu", "tf_mlp.cu"])
def test_copies_to_the_device_are_stream_ordered(name):
    code = _code(name)
    plain = [m.start() for m in re.finditer(r"\bcudaMemcpy\s*\(", code)]
    assert not plain, [code[p:p + 80] for p in plain]
    for m in re.finditer(r"\bcudaMemcpyToSymbol\s*\(", code):     # on the legacy stream: waited for
        rest = code[m.end():]
        body = rest[:rest.index("return TF_OK")]
        assert "cudaStreamSynchronize(cudaStreamLegacy)" in body, code[m.start():m.start() + 80]
