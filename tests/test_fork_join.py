"""The second stream of a right-hand side is joined whatever way the call ends
(csrc/ih_fork.cuh), compiled for the host against a fake runtime that records
the calls and fails on demand."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "instaheat_gb300" / "csrc"

FAKE = """
#pragma once
#include <cstdio>
typedef int cudaError_t;
typedef const char *cudaStream_t;
typedef const char *cudaEvent_t;
constexpr int cudaSuccess = 0;
extern int fail_at, calls;
inline int count() { return ++calls == fail_at ? 719 : 0; }
inline int cudaEventRecord(cudaEvent_t e, cudaStream_t s) { printf("record %s %s\\n", e, s); return count(); }
inline int cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, int) { printf("wait %s %s\\n", s, e); return count(); }
"""

MAIN = """
#include <cstdlib>
#include "ih_fork.cuh"
int fail_at = 0, calls = 0;
// a call that forks, launches on both streams and may fail in between
static int body(bool fork, int launch_fails) {
  ih::Fork f;
  if (fork) {
    int e = f.start("main", "side", "begin", "end");
    if (e) return e;
  }
  for (int i = 1; i <= 3; ++i) {
    if (i == launch_fails) return 700 + i;
    printf("launch %d\\n", i);
  }
  int e = f.join();
  if (e) return e;
  printf("after\\n");
  return 0;
}
int main(int argc, char **argv) {
  fail_at = atoi(argv[3]);
  int r = body(atoi(argv[1]), atoi(argv[2]));
  printf("status %d\\n", r);
  return 0;
}
"""


def test_every_exit_joins(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", str(CSRC),
                    str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)

    def run(fork, launch_fails=0, fail_at=0):
        out = subprocess.run([str(exe), str(int(fork)), str(launch_fails), str(fail_at)],
                             check=True, capture_output=True, text=True).stdout.split("\n")
        return out[:-1]

    begin = ["record begin main", "wait side begin"]
    end = ["record end side", "wait main end"]
    launches = ["launch 1", "launch 2", "launch 3"]
    assert run(True) == begin + launches + end + ["after", "status 0"]
    assert run(False) == launches + ["after", "status 0"]
    for i in (1, 2, 3):  # a launch fails: joined, once, before the call returns
        assert run(True, i) == begin + launches[:i - 1] + end + ["status %d" % (700 + i)]
        assert run(False, i) == launches[:i - 1] + ["status %d" % (700 + i)]
    # the fork itself fails: nothing runs on the second stream, nothing to join
    assert run(True, 0, 1) == begin[:1] + ["status 719"]
    assert run(True, 0, 2) == begin + ["status 719"]
    # the join's own calls fail: reported, not repeated
    assert run(True, 0, 3) == begin + launches + end[:1] + ["status 719"]
    assert run(True, 0, 4) == begin + launches + end + ["status 719"]


def test_right_hand_side_uses_it():
    src = (CSRC / "ih_rhs.cu").read_text()
    assert "Fork beside;" in src and "beside.join()" in src
    assert "cudaStreamWaitEvent(c->side" not in src  # no fork of its own
