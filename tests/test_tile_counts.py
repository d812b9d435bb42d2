"""How the CTAs of the summing pack kernel share the tile counts with the one that overwrites them
(cswap_b200/csrc/tile_counts.cuh), on the CPU with threads for CTAs, under the compiler's race detector."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_counts_are_overwritten_behind_all_reads(tmp_path):
    exe = str(tmp_path / "race")
    build = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=thread", "-pthread", "-o", exe,
                            os.path.join(HERE, "tile_counts_race.cpp")], capture_output=True, text=True)
    if "libtsan" in build.stderr or "fsanitize" in build.stderr:
        pytest.skip("the compiler has no race detector")
    assert build.returncode == 0, build.stderr
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    if "unexpected memory mapping" in run.stderr:
        pytest.skip("the race detector cannot place its memory here")
    assert run.returncode == 0, run.stderr[:4000]
