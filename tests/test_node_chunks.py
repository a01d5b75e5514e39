"""Nodes handed out in chunks, up to the largest grids (node_chunk.h)."""

import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_last_chunks(tmp_path):
    exe = str(tmp_path / "node_chunk_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "cpp", "node_chunk_check.cpp")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
