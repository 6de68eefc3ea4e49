"""The dense eigensolver's second stream is joined however the call ends: an early return must not leave its kernels
writing the context's workspace behind the next call's back.  The guard is compiled against recording stand-ins for
the CUDA calls; no GPU is needed."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bsr_b200", "csrc")

FAKE = """
#pragma once
#include <string>
typedef const char *cudaStream_t;
typedef const char *cudaEvent_t;
typedef int cudaError_t;
constexpr int cudaSuccess = 0;
extern std::string calls;
extern int record_error;
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { calls += std::string("record ") + e + " on " + s + ";"; return record_error; }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { calls += std::string(s) + " waits for " + e + ";"; return 0; }
"""

MAIN = """
#include <cstdio>
#include <cstring>
#include "aux_join.h"
std::string calls;
int record_error = 0;
static int solve(const char *aux, int leave_at)
{
    bsrg::AuxJoin join(aux, "main", "event");
    if (leave_at == 0) return 1;
    calls += "work;";
    if (leave_at == 1) return 1;
    calls += "joined;";
    join.done();
    return 0;
}
int main(int argc, char **argv)
{
    record_error = atoi(argv[3]);
    solve(strcmp(argv[1], "none") ? argv[1] : nullptr, atoi(argv[2]));
    printf("%s", calls.c_str());
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("aux_join")
    (d / "cuda_runtime.h").write_text(FAKE)
    (d / "main.cpp").write_text("#include <cstdlib>\n" + MAIN)
    exe = str(d / "main")
    subprocess.run(["g++", "-std=c++17", "-I", str(d), "-I", CSRC, str(d / "main.cpp"), "-o", exe], check=True)
    return lambda *a: subprocess.run([exe] + [str(x) for x in a], check=True, capture_output=True, text=True).stdout


@pytest.mark.parametrize("aux,leave_at,error,calls", [
    ("aux", 0, 0, "record event on aux;main waits for event;"),
    ("aux", 1, 0, "work;record event on aux;main waits for event;"),
    ("aux", 2, 0, "work;joined;"),
    ("aux", 1, 1, "work;record event on aux;"),             # nothing was recorded: nothing to wait for
    ("none", 1, 0, "work;"),                                # no second stream
])
def test_guard(program, aux, leave_at, error, calls):
    assert program(aux, leave_at, error) == calls


def test_the_solver_is_guarded():
    """The guard stands before the first call that queues work on the second stream."""
    src = open(os.path.join(CSRC, "syevd2.cu")).read()
    body = src[src.index("static int syevd2_impl("):src.index("\nint dense_syevd(")]
    at = body.index("AuxJoin ")
    assert at < body.index("sy2sb(") and at < body.index("q1_tfactors(")
