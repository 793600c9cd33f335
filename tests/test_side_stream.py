"""Work beside the main stream (csrc/side.h): whatever way a call leaves the scope that forked it, the main stream has
to wait for the side stream, or the next call writes buffers that the side stream still reads.  The header is compiled
against a fake CUDA runtime that writes down the calls, each of which can be told to fail."""
import glob
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ornith-rs_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "side.h"
static const char* fails = "";
static cudaError_t said(const char* what, const void* a, const void* b) {
  printf("%s %c%c;", what, a ? (char)(size_t)a : '-', b ? (char)(size_t)b : '-');
  return strstr(fails, what) ? cudaErrorUnknown : cudaSuccess;
}
extern "C" {
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return said("record", e, s); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { return said("wait", s, e); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return said("sync", s, nullptr); }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
int call(int leave, bool two) {
  SideWork w((cudaStream_t)'M', two ? (cudaStream_t)'S' : nullptr, (cudaEvent_t)'f', (cudaEvent_t)'j');
  if (w.mark() != cudaSuccess || leave == 0) return 1;
  if (w.start() != cudaSuccess) return 1;
  printf("work %c;", (char)(size_t)w.stream());
  if (leave == 1) return 1;
  if (w.done() != cudaSuccess || leave == 2) return 1;
  if (w.join() != cudaSuccess) return 1;
  return 0;
}
int main(int, char** v) {
  fails = v[3];
  const int rc = call(atoi(v[1]), v[2][0] == '2');
  printf("end %d", rc);
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("side")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", CUDA + "/include", str(d / "h.cpp"), "-o", str(d / "h")], check=True)
    return lambda leave, streams, fails="": subprocess.run([str(d / "h"), str(leave), str(streams), fails], check=True,
                                                           capture_output=True, text=True).stdout


def test_an_ordinary_call_forks_and_joins_once(harness):
    assert harness(9, 2) == "record fM;wait Sf;work S;record jS;wait Mj;end 0"
    assert harness(9, 1) == "work M;end 0"


@pytest.mark.parametrize("leave,fails", [(1, ""), (2, ""), (9, "record"), (9, "wait")])
def test_a_call_that_leaves_early_joins_all_the_same(harness, leave, fails):
    """After the last piece of work the main stream waits for the side stream, or the host does."""
    log = harness(leave, 2, fails)
    assert log.endswith("end 1")
    if "wait S" in log:      # the side stream was given (or could have been given) work
        tail = log[log.rindex("wait S"):]
        assert re.search(r"record jS;wait Mj;", tail) and not fails or "sync S" in tail, log


def test_nothing_to_join_before_the_fork(harness):
    assert harness(0, 2) == "record fM;end 1"


def test_every_fork_goes_through_it():
    """No file records or waits for the context's fork and join events itself."""
    used = {os.path.basename(f): re.findall(r"cuda(?:EventRecord|StreamWaitEvent)\([^;]*(?:ev_fork|ev_join|->side)", open(f).read())
            for f in glob.glob(os.path.join(CSRC, "*.cu*"))}
    assert not {f: u for f, u in used.items() if u}
    src = {f: open(os.path.join(CSRC, f)).read() for f in ("model.cu", "batch.cu", "ep.cu")}
    assert [src[f].count("orn_side_work(") for f in src] == [2, 1, 1]
