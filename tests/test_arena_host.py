"""DevArena (csrc/device/arena.hpp) compiled against counted stand-ins of the
runtime's allocation calls (tests/cxx/fake_cuda): buffers with memory of their
own are freed when released, also at the size of a chunk, and a dry arena
counts what a real one takes."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_arena(tmp_path):
    exe = str(tmp_path / "arena_test")
    cxx = os.path.join(ROOT, "tests", "cxx")
    cmd = ["g++", "-std=c++17", "-O1", "-I" + os.path.join(cxx, "fake_cuda"),
           "-I" + os.path.join(ROOT, "hfls_b200", "csrc", "device"), os.path.join(cxx, "arena_test.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "arena ok\n", r.stdout + r.stderr
