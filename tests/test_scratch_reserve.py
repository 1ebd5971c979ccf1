"""The scratch of an evaluation lies in one allocation (DevBufSet of
csrc/qb_engine.h).  An allocation that fails must leave nothing behind: the next
reservation asks for its own sizes alone.  A small host program linked to the
library makes the allocation fail (2^60 bytes; without a GPU every allocation
fails) and looks at what the next one asks for; with a GPU that one succeeds.
"""
import os
import shutil
import subprocess

import pytest

import qbgpu
from conftest import REPO

PROGRAM = r"""
#include <cstdio>
#include "qb_engine.h"
int main() {
	int devices = 0;
	if (cudaGetDeviceCount(&devices) != cudaSuccess) devices = 0;
	cudaGetLastError();
	qb::DevBuf a, b, c;
	qb::DevBufSet set;
	auto fails = [&] {
		try { set.reserve(); } catch (const std::exception &) { return true; }
		return false;
	};
	set.add(a, (size_t)1 << 60);
	set.add(b, 512);
	if (!fails() || !set.want.empty() || a.p || b.p) return 1;
	set.add(b, 1000);
	set.add(c, 300);
	set.add(b, 700);                       // twice the same buffer: the larger size
	if (set.want.size() != 2 || set.want[0].second != 1000) return 2;
	const bool failed = fails();
	if (!set.want.empty()) return 3;
	if (devices == 0) return failed ? 0 : 4;
	if (failed) return 5;
	if (set.whole.bytes != 1024 + 512 || b.bytes != 1024 || c.bytes != 512) return 6;
	set.add(a, 256);                       // growth: the earlier buffers move along
	set.reserve();
	if (set.whole.bytes != 256 + 1024 + 512 || !a.p || !b.p || !c.p) return 7;
	std::puts("reserved");
	return 0;
}
"""


def run_program(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    pkg = os.path.dirname(os.path.abspath(qbgpu.__file__))
    src, exe = tmp_path / "reserve.cc", tmp_path / "reserve"
    src.write_text(PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    r = subprocess.run(["g++", "-std=c++17", "-O1", str(src), "-o", str(exe), "-I", os.path.join(pkg, "csrc"), "-I", os.path.join(REPO, "include"),
                        "-I", os.path.join(cuda, "include"), "-L", os.path.join(pkg, "lib"), "-l:libqbgpu.so", "-L", os.path.join(cuda, "lib64"),
                        "-lcudart", "-Wl,-rpath," + os.path.join(pkg, "lib") + ":" + os.path.join(cuda, "lib64")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, env=dict(os.environ, QB_ABORT_ON_ERROR="0"))
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    return r.stdout


def test_failed_reservation_leaves_nothing_behind(tmp_path):
    run_program(tmp_path)


@pytest.mark.gpu
def test_reservation_after_a_failed_one(tmp_path):
    assert run_program(tmp_path).strip() == "reserved"
