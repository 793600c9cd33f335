"""The library works on streams of its own that do not wait for the legacy default stream, so device memory that
its kernels read must not be prepared there: a clear or a copy without a stream is allowed only where the same
expression waits for the device behind it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ornith-rs_b200", "csrc")


def legacy_calls(src):
    """Statements with a clear or copy that names no stream and no wait."""
    src = re.sub(r"//[^\n]*", "", src)
    return [st.strip() for st in re.split(r"[;{}]", src)
            if re.search(r"\bcudaMem(set|cpy|cpy2D|set2D)\(", st) and "cudaDeviceSynchronize()" not in st]


def test_nothing_is_prepared_on_the_legacy_stream():
    found = {os.path.basename(f): legacy_calls(open(f).read()) for f in glob.glob(os.path.join(CSRC, "*.cu*"))}
    assert not {f: c for f, c in found.items() if c}


def test_the_check_sees_a_clear_without_a_stream():
    assert legacy_calls("int f() { CK(cudaMemset(p, 0, 4)); }")
    assert not legacy_calls("int f() { ok = cudaMemset(p, 0, 4) == 0 && cudaDeviceSynchronize() == 0; }")
    assert not legacy_calls("int f() { CK(cudaMemsetAsync(p, 0, 4, s)); }  // cudaMemset(p)")
