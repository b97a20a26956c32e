"""CPU: the torch binding as a module: what it is linked with."""
import os
import subprocess

from conftest import ROOT

NATIVE = os.path.join(ROOT, "tinytorch_b200", "lib", "_native.so")


def test_one_libstdcxx_in_the_process():
    if not os.path.exists(NATIVE):
        from tinytorch_b200.build import build_native
        build_native()
    needed = subprocess.run(["ldd", NATIVE], capture_output=True, text=True, check=True).stdout
    assert "libstdc++.so.6" in needed
