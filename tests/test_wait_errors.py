"""A wait that makes kernels' results visible to the host also looks at the
context's error word (sync_checked in csrc/common.cuh), checked without a GPU:
the helper itself, compiled with g++ against a fake CUDA runtime, and that no
entry point waits for a stream without it. The kernels' own bounded waits
(csrc/wait.cuh) run on the host the same way."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lambda_vm_b200", "csrc")
CHOST = os.path.join(ROOT, "tests", "c_host")

# Plain waits: the helper's own, those that only drain streams (after a failure,
# or before the checked wait on the caller's stream), and the root table's,
# whose kernel waits for nothing.
PLAIN = {
    "common.cuh": ["cudaError_t e = cudaStreamSynchronize(st);"],
    "api.cu": ["if (cs && rc != SG_OK) cudaStreamSynchronize(cs);",
               'if (streams[s]) cuda_ok(cudaStreamSynchronize(streams[s]), "sync");',
               "cudaStreamSynchronize(streams[s]);",
               "if (rc != SG_OK) cudaStreamSynchronize(streams[s]);",
               "cudaStreamSynchronize(st);"],
    "ntt.cu": ["SG_CUDA(cudaStreamSynchronize(st));"],
}


def test_waits_go_through_the_checked_helper():
    for fn in sorted(os.listdir(CSRC)):
        src = open(os.path.join(CSRC, fn)).read()
        lines = [l.strip() for l in src.split("\n") if "cudaStreamSynchronize(" in l]
        assert lines == PLAIN.get(fn, []), fn
    used = sum(len(re.findall(r"\bsync_checked\(", open(os.path.join(CSRC, f)).read())) for f in os.listdir(CSRC))
    assert used >= 19


# wait_errors: the helper; bounded_wait: a kernel's wait gives up at its limit,
# and at once behind another's timeout
@pytest.mark.parametrize("program", ["wait_errors", "bounded_wait"])
def test_host_programs(tmp_path, program):
    exe = str(tmp_path / program)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(CHOST, "fake_cuda"),
                        "-I" + os.path.join(ROOT, "include"), os.path.join(CHOST, program + ".cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    run = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stdout + run.stderr
