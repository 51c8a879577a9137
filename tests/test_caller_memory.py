"""The rules by which a call works in the caller's own device memory (csrc/caller_memory.cuh), through
tests/cpp/caller_memory.cpp: plain values, so memory of another GPU is covered without one."""
import os
import subprocess

CPP = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp")


def test_rules_on_plain_values():
    subprocess.run(["make", "-s", "-C", CPP, "_build/caller_memory"], check=True)
    r = subprocess.run([os.path.join(CPP, "_build", "caller_memory")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
