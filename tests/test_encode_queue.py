"""The 3-D encoder's expansion queue, on the CPU: what a step needs of it has been read a step before, within its slots."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_entries_are_read_ahead(tmp_path):
    exe = str(tmp_path / "queue")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wno-unknown-pragmas", "-o", exe,
                           os.path.join(HERE, "encode_queue.cpp")])
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr
