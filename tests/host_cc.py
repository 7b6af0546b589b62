"""Compile a small C++ program against the library's host headers and run it (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

from rockseis_b200 import build


def run_cpp(tmp_path, code, sources=(), flags=("-O1",)):
    """Output of the program `code`, linked with the csrc files named in `sources`."""
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    main, exe = tmp_path / "main.cpp", tmp_path / "main"
    main.write_text(code)
    cmd = ["g++", "-std=c++17", "-ffp-contract=off", *flags, "-I" + build.CSRC, "-I" + build.INCLUDE, "-I" + cuda, str(main),
           *[os.path.join(build.CSRC, s) for s in sources], "-o", str(exe), "-lpthread"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
