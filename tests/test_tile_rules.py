"""Host-side rules of the launches (which devices a number is kept for, what a launch costs on the host, how the
fp32 kernels are split), as small programs built with the kernels' own headers and run on the CPU."""
import importlib
import os
import subprocess

import pytest

build = importlib.import_module("610sample_b200._build")
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("rules", ["tile_rules", "split_rules"])
def test_rules_hold_on_the_host(tmp_path, rules):
    if not os.path.exists(build._nvcc()):
        pytest.skip("no nvcc")
    program = str(tmp_path / rules)
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-cudart", "shared", os.path.join(HERE, "host", rules + ".cu"), "-o", program], check=True)
    libs = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "lib64")
    env = dict(os.environ, LD_LIBRARY_PATH=libs + os.pathsep + os.environ.get("LD_LIBRARY_PATH", ""))
    done = subprocess.run([program], capture_output=True, text=True, timeout=60, env=env)
    assert done.returncode == 0, done.stdout + done.stderr
