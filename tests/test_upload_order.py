"""Uploads come before the kernels that read them.

cudaMemcpy and cudaMemcpyToSymbol may return once pageable host data is staged,
before it is on the device, and the library's streams are non-blocking: they do
not wait for the default stream.  So an upload goes to the stream of the kernels
that read it, or is waited for.  It shows on a busy device only, hence this
reads the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qsl_gb300", "csrc")


def test_uploads_on_the_default_stream_are_waited_for():
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        code = re.sub(r"#ifdef QSLC_DEBUG_BOUNDS.*?#endif", "", code, flags=re.S)   # debug builds synchronise the device
        for m in re.finditer(r"\bcudaMemcpy(?:ToSymbol)?\(", code):
            body = code[m.start():]
            body = body[:body.index("\n}")]              # to the end of the function
            assert "cudaStreamSynchronize(cudaStreamLegacy)" in body, (name, body.split("\n")[0])
