"""Host sources of the library on the CPU: C++ programs under tests/host,
compiled with them and a CUDA runtime in host memory (tests/host/fake_cuda.h)."""

import pathlib
import shutil
import subprocess

from psycles_b200 import build

HOST = pathlib.Path(__file__).resolve().parent / "host"


def run(name, tmp_path, *sources):
    exe = tmp_path / name
    subprocess.run([shutil.which("g++"), *build.CXX_FLAGS, f"-I{build.CUDA_HOME / 'include'}",
                    str(HOST / f"{name}.cpp"), *(str(build.CSRC / s) for s in sources), "-lpthread",
                    # launches and entry points that the program does not reach
                    "-Wl,--unresolved-symbols=ignore-all", "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)


def test_edits_rejected_for_memory_leave_the_scene_as_it_was(tmp_path):
    r = run("versioned_edit", tmp_path, "psy_host.cpp", "psy_light_tree.cpp")
    assert r.returncode == 0, r.stdout + r.stderr


def test_byte_boxes_against_float_boxes(tmp_path):
    r = run("node_boxes", tmp_path, "psy_light_tree.cpp")
    assert r.returncode == 0, r.stdout + r.stderr
