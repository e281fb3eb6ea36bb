"""A source-level invariant of the host code that no compiler checks.

The library's own streams are non-blocking, so they do not wait for the default stream, and cudaMemcpy from pageable or
device memory and cudaMemset may return before the default stream has done the work.  Load-time copies therefore go
through upload_now / clear_now (csrc/api.cu), which wait for it; everything else is an ...Async call on the stream of
its use.
"""
import re
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "apus-deepseek-v4-flash_b200" / "csrc"


def body(text, head):
    k = text.index(head)
    return text[k:text.index("\n}", k)]


def test_no_copy_or_clear_on_the_default_stream_without_a_wait():
    api = (SRC / "api.cu").read_text()
    inside = body(api, "int upload_now(") + body(api, "int clear_now(")
    assert inside.count("cudaStreamSynchronize(cudaStreamLegacy)") == 2
    found = []
    for f in sorted(SRC.glob("*.cu")) + sorted(SRC.glob("*.cuh")):
        for line in f.read_text().splitlines():
            code = line.split("//")[0]
            if re.search(r"\bcuda(Memcpy|Memset|Memcpy2D)\s*\(", code) and line not in inside:
                found.append(f"{f.name}: {line.strip()}")
    assert not found, found
