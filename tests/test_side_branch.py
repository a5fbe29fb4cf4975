"""SideBranch (csrc/hm_branch.h), which forks a frame's shadow rays off to a
second stream: the order of its calls, and that a branch left open by an early
return is joined.  Compiled for the host against a fake of the three runtime
calls, which records them and fails the one it is told to."""
import os
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "hairmsnn_gb300" / "csrc"
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "hm_branch.h"
static int calls = 0, fail_at = -1;
static cudaError_t note(const char* what) {
  const bool bad = calls++ == fail_at;
  printf("%s%s ", what, bad ? "!" : "");
  return bad ? cudaErrorInvalidValue : cudaSuccess;
}
static const char* name(const void* s) { return s == (void*)1 ? "main" : "side"; }
extern "C" cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  char b[32];
  snprintf(b, sizeof(b), "rec%ld@%s", (long)e, name(s));
  return note(b);
}
extern "C" cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  char b[32];
  snprintf(b, sizeof(b), "%s<%ld", name(s), (long)e);
  return note(b);
}
extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  char b[32];
  snprintf(b, sizeof(b), "sync@%s", name(s));
  return note(b);
}
// rounds of fork / end / join; leaves early after `steps` calls of SideBranch
static int run(int rounds, int steps, bool one_stream) {
  hm::SideBranch b((cudaStream_t)1, (cudaStream_t)(one_stream ? 1 : 2), (cudaEvent_t)1, (cudaEvent_t)2);
  for (int i = 0; i < rounds; ++i) {
    if (steps-- == 0) return 1;
    if (b.join() != cudaSuccess) return 2;
    if (steps-- == 0) return 1;
    if (b.fork() != cudaSuccess) return 2;
    if (steps-- == 0) return 1;
    if (b.end() != cudaSuccess) return 2;
  }
  return b.join() != cudaSuccess ? 2 : 0;
}
int main(int, char** a) {
  fail_at = atoi(a[4]);
  const int r = run(atoi(a[1]), atoi(a[2]), atoi(a[3]));
  printf("-> %d\n", r);
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if not (CUDA / "cuda_runtime_api.h").is_file():
        pytest.skip("no CUDA headers")
    d = tmp_path_factory.mktemp("branch")
    (d / "b.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-I", str(CUDA), str(d / "b.cpp"), "-o", str(d / "b")],
                   check=True)

    def call(rounds, steps=-1, one_stream=0, fail_at=-1):
        return subprocess.run([str(d / "b"), str(rounds), str(steps), str(one_stream), str(fail_at)], check=True,
                              capture_output=True, text=True).stdout.strip()
    return call


FORK, END, JOIN = "rec1@main side<1 ", "rec2@side ", "main<2 "


def test_order(run):
    assert run(2) == FORK + END + JOIN + FORK + END + JOIN + "-> 0"
    assert run(3, one_stream=1) == "-> 0"
    assert run(0) == "-> 0"


@pytest.mark.parametrize("steps,before", [(0, ""), (1, ""), (2, FORK), (3, FORK + END), (4, FORK + END + JOIN),
                                          (5, FORK + END + JOIN + FORK)])
def test_early_return_joins_an_open_branch(run, steps, before):
    still_open = before.count("side<1") > before.count("main<2")
    assert run(2, steps) == before + (END + JOIN if still_open else "") + "-> 1"


def test_failed_calls_are_returned(run):
    assert run(1, fail_at=0) == "rec1@main! -> 2"  # nothing on the side stream yet
    assert run(1, fail_at=1) == "rec1@main side<1! -> 2"
    assert run(1, fail_at=2) == FORK + "rec2@side! " + END + JOIN + "-> 2"
    assert run(1, fail_at=3) == FORK + END + "main<2! " + END + JOIN + "-> 2"


def test_branch_that_cannot_be_joined_is_waited_for(run):
    assert run(1, steps=2, fail_at=2) == FORK + "rec2@side! sync@side -> 1"
