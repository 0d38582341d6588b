"""The engine's host arrays reach the device before anything reads them: its own stream is not ordered
behind the default stream, and a copy of pageable memory there may return before it has landed, so
every upload is issued on a named stream and waited for (phx_upload, phx_upload_rows)."""
import os
import re

from tests.conftest import ROOT

ENGINE = os.path.join(ROOT, "opticks_b200", "csrc", "phx_engine.cu")


def _code():
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", open(ENGINE).read(), flags=re.S)


def test_no_copy_on_the_default_stream():
    code = _code()
    assert not re.findall(r"\bcudaMem(?:cpy|cpy2D|cpy2DToArray|cpyToSymbol|set)\s*\(", code)


def test_creation_uploads_are_waited_for():
    code = _code()
    for fn in ("phx_upload", "phx_upload_rows"):
        body = re.search(r"static cudaError_t %s\(.*?\n}" % fn, code, flags=re.S).group(0)
        assert "Async(" in body and "cudaStreamSynchronize(st)" in body
    create = re.search(r"\nint phx_create\(.*?\n}", code, flags=re.S).group(0)
    assert len(re.findall(r"\bphx_upload\(", create)) >= 11
    assert not re.search(r"\bcudaMemcpy\w*\(", create)
