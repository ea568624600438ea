"""The side streams of the eigensolver are joined on every way out of a call (CPU, with fakes of the CUDA
calls)."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "nrgljubljana_b200", "csrc")


def test_joined_on_every_way_out(tmp_path):
    exe = str(tmp_path / "side_streams")
    r = subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include",
                        os.path.join(ROOT, "tests", "cpp", "side_streams_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and "SIDE STREAMS OK" in r.stdout, r.stdout


def test_side_streams_are_registered_where_they_fork():
    """In the solver's launches, every stream that is made to wait for a fork event is handed to SideStreams
    in the next statement, so that no return in between leaves it unjoined."""
    src = open(os.path.join(CSRC, "eig_large.cu")).read()
    forks = re.findall(r"cudaStreamWaitEvent\((?:ss|c->side3), c->\w*fork\w*, 0\)\);\s*(?:s3 = c->side3;\s*)?(\w+\.add)?", src)
    assert len(forks) == 2 and all(forks)
