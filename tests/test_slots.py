"""The slots of row vectors in shared memory (weavess_gb300/csrc/wv_slots.cuh):
no slot is taken while a copy into it may be under way."""
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_slot_is_taken_with_a_copy_under_way():
    with tempfile.TemporaryDirectory() as tmp:
        exe = os.path.join(tmp, "chk")
        subprocess.check_call(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "native", "slots_check.cpp")])
        out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
        assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout + out.stderr
