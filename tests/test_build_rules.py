"""The Makefile's dependencies on headers (dry runs on a copy with empty objects)."""
import os
import shutil
import subprocess
import time

import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "simplex-benchmarks_b200")


def commands(tree):
    r = subprocess.run(["make", "-n", "-C", str(tree / "pkg")], capture_output=True, text=True, check=True)
    return r.stdout


def age(path, t):
    os.utime(path, (t, t))


@pytest.mark.parametrize("listed", [False, True])
def test_header_change_rebuilds(tmp_path, listed):
    """Objects without a header list (from rules that wrote none) follow every header,
    objects with one follow it."""
    shutil.copytree(os.path.join(PKG, "csrc"), tmp_path / "pkg" / "csrc")
    shutil.copytree(os.path.join(os.path.dirname(PKG), "include"), tmp_path / "include")
    shutil.copy(os.path.join(PKG, "Makefile"), tmp_path / "pkg")
    build = tmp_path / "pkg" / "_build"
    build.mkdir()
    t = time.time() - 1000
    for d, _, files in os.walk(tmp_path):
        for f in files:
            age(os.path.join(d, f), t)
    names = [os.path.splitext(f)[0] for f in os.listdir(tmp_path / "pkg" / "csrc") if f.endswith((".cu", ".cpp"))]
    for n in names:
        (build / (n + ".o")).touch()
        age(build / (n + ".o"), t + 100)
        if listed:
            header = "csrc/operator.hpp" if n in ("capi", "operator") else "csrc/mesh.hpp"
            (build / (n + ".d")).write_text(f"_build/{n}.o: {header}\n")
    (tmp_path / "pkg" / "libsimplexfem.so").touch()
    age(tmp_path / "pkg" / "libsimplexfem.so", t + 100)
    assert "-c csrc/" not in commands(tmp_path)
    age(tmp_path / "pkg" / "csrc" / "operator.hpp", t + 200)
    out = commands(tmp_path)
    rebuilt = {n for n in names if f"-o _build/{n}.o" in out}
    assert rebuilt == ({"capi", "operator"} if listed else set(names))
