"""Source-level invariants of the bounded waits that no compiler checks: one status word, read with one copy."""
import re
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "apus-deepseek-v4-flash_b200" / "csrc"
TEXT = {f.name: f.read_text() for f in sorted(SRC.glob("*.cu")) + sorted(SRC.glob("*.cuh"))}


def test_the_status_of_the_waits_is_read_with_one_copy():
    """It is read behind every forward, each copy a blocking round trip."""
    reads = [n for n, t in TEXT.items() for _ in re.finditer(r"\bcudaMemcpyFromSymbol\s*\(", t)]
    assert reads == ["api.cu"], reads


def test_every_kernel_that_waits_records_into_that_word():
    for name, t in TEXT.items():
        for m in re.finditer(r"atomicCAS\(([^,]+),\s*0,\s*(fail|31)\)", t):
            assert m.group(1) in ("a.status", "status"), (name, m.group(0))
