"""The nodes of one local-join launch (weavess_gb300/csrc/wv_join_plan.h): its
offers and its list entries stay within what a launch may hold."""
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))


def test_join_chunks_stay_within_their_limits():
    with tempfile.TemporaryDirectory() as tmp:
        exe = os.path.join(tmp, "chk")
        subprocess.check_call(["g++", "-O2", "-std=c++17", "-o", exe,
                               os.path.join(HERE, "native", "join_plan_check.cpp")])
        out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
        assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout + out.stderr
