"""Host-side rules of the tensor-core launches (which devices a number is kept for, what a launch costs on the
host), as a small program built with the kernels' own header and run on the CPU."""
import importlib
import os
import subprocess

import pytest

build = importlib.import_module("610sample_b200._build")
HERE = os.path.dirname(os.path.abspath(__file__))


def test_rules_hold_on_the_host(tmp_path):
    if not os.path.exists(build._nvcc()):
        pytest.skip("no nvcc")
    program = str(tmp_path / "tile_rules")
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-cudart", "shared", os.path.join(HERE, "host", "tile_rules.cu"), "-o", program], check=True)
    libs = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "lib64")
    env = dict(os.environ, LD_LIBRARY_PATH=libs + os.pathsep + os.environ.get("LD_LIBRARY_PATH", ""))
    done = subprocess.run([program], capture_output=True, text=True, timeout=60, env=env)
    assert done.returncode == 0, done.stdout + done.stderr
