"""The host's read-back after a step with norms (csrc/norms_read.h) against a stream whose
copies and kernel writes arrive only when it is waited for, which is all that CUDA promises
for an asynchronous copy into pageable memory."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(__file__)), "cvfes_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>
#include "norms_read.h"

struct LateStream {  // everything queued happens at wait()
    std::vector<std::function<void()>> queue;
    int cleared = 0;
    int copy(void* d, const void* s, unsigned long long n) {
        queue.push_back([=] { std::memcpy(d, s, n); });
        return 0;
    }
    int wait() {
        for (auto& f : queue) f();
        queue.clear();
        return 0;
    }
    int clear(int32_t* p) { ++cleared; *p = 0; return 0; }
};

int main(int argc, char** argv) {
    const bool direct = std::atoi(argv[1]);
    int32_t status = std::atoi(argv[2]);
    const double count = std::atof(argv[3]);
    double dev[8] = {1, 2, 3, 0, 5, 6, 7, count}, host[8] = {0};
    LateStream st;
    if (direct) st.queue.push_back([&] { std::memcpy(host, dev, sizeof(dev)); });  // the kernel
    cvfes::StepReadBack r;
    const int rc = cvfes::read_step_norms(st, host, direct ? nullptr : dev, 2, &status, r);
    std::printf("%d %d %g %d %d %g\n", rc, r.status, r.nonfinite, st.cleared, (int)st.queue.size(),
                host[0] + host[7]);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("norms_read")
    (d / "main.cpp").write_text(PROGRAM)
    exe = str(d / "main")
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-I", CSRC, str(d / "main.cpp"),
                    "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("direct", [0, 1])
@pytest.mark.parametrize("status", [0, 1])
@pytest.mark.parametrize("count", [0, 3])
def test_nothing_is_read_before_the_stream_was_waited_for(program, direct, status, count):
    out = subprocess.run([program, str(direct), str(status), str(count)], check=True,
                         capture_output=True, text=True).stdout.split()
    assert out == ["0", str(status), str(count), str(status), "0", str(1 + count)]
