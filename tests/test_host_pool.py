"""The pool of a server's request buffers: a first request is served from it, freed room is good
for requests of any size, its bound, and what it does without page-locked memory."""
import subprocess

from bonxai_gb300 import build as B
from conftest import ROOT


def test_host_pool(tmp_path):
    exe = tmp_path / "host_pool"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", f"-I{B.CSRC}", "-o", str(exe),
                    str(ROOT / "tests" / "cpp" / "host_pool_main.cpp"), "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
