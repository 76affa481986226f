"""Uploads from host memory go through the context's stream.  That stream is non-blocking: a plain
cudaMemcpy (legacy stream, and from pageable memory possibly still in flight when it returns) would not be
ordered before the kernels that read the data."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "blamm_gb300", "csrc", "blamm_gpu.cu")


def test_no_upload_on_the_legacy_stream():
    text = open(SRC).read()
    calls = re.findall(r"\bcudaMemcpy\s*\([^;]*cudaMemcpyHostToDevice[^;]*;", text)
    assert not calls, calls
    assert not re.findall(r"\bcudaMemset\s*\(", text)
    for call in re.findall(r"\bcudaMemcpyAsync\s*\([^;]*cudaMemcpyHostToDevice[^;]*;", text):
        assert "ctx->stream" in call or "ctx->copy_stream" in call, call
