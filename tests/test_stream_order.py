"""The library works on streams of its own that do not wait for the legacy default stream, so device memory that
its kernels read must not be prepared there: a clear or a copy without a stream is allowed only where the same
expression waits for the device behind it."""
import glob
import os
import re

import pytest

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


def refills(body, read, issue):
    """The refills of a loop body's ring in two passes over it, each with whether a barrier stands between the warp's
    last read and it."""
    out, read_since = [], False
    for m in list(re.finditer(r"(?P<sync>__sync(warp|threads)\(\))|(?P<read>%s)|(?P<issue>%s)" % (read, issue), re.sub(r"//[^\n]*", "", body))) * 2:
        if m["sync"]:
            read_since = False
        elif m["read"]:
            read_since = True
        else:
            out.append(not read_since)
    return out


@pytest.mark.parametrize("name,kernel,loop,read,issue,refilled", [
    ("batch.cu", "battn_partial_kernel(", "for (int i = 0; i < my_tiles; ++i) {", r"ldsm4t?\((?:ks|vs)\b", r"\bissue\(", 4),
    ("flash.cu", "flash_prefill_kernel(", "for (int i = 0; i < tiles; ++i) {", r"ldsm4t?\((?:kt|vs)\b", r"\bissue\(", 2),
    ("gdn_chunk.cu", "gdn_chunk_scan_kernel(", "for (int c = 0; c < p.nchunks; ++c) {", r"ldsm4t?\((?:kg|qg|tm|pm|kd)\b|\(vptr", r"\bissue\(", 2),
])
def test_a_place_is_refilled_behind_a_barrier(name, kernel, loop, read, issue, refilled):
    """The rings that cp.async fills: between a warp's last read of a place and the copy that refills it stands a barrier,
    since shuffles and votes order no memory accesses."""
    src = open(os.path.join(CSRC, name)).read()
    src = src[src.index(kernel):]
    src = src[src.index(loop):]
    got = refills(src[:src.index("\n  }\n")], read, issue)
    assert got == [True] * refilled, got
