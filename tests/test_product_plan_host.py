"""The plans of the tensor core products where the number of SMs is not known (no device, or one that does not answer)."""
import os
import subprocess
import sys

PROBE = """
import ctypes, sys
from llm_singularity_b200.kernels import build
lib = ctypes.CDLL(build.ensure_built(["gemm_tc"])["gemm_tc"])
swap, bn, splits = (ctypes.c_int() for _ in range(3))
for M in (1, 64, 129, 257, 2048, 70000):
    for N in (1, 64, 128, 1000, 28672):
        for K in (8, 512, 14336):
            for gated in (0, 1):
                rc = lib.lsb_gemm_tc_plan(M, N, K, gated, ctypes.byref(swap), ctypes.byref(bn), ctypes.byref(splits))
                assert rc == 0 and 16 <= bn.value <= 256 and 1 <= splits.value <= 8, (M, N, K, gated, bn.value, splits.value)
                assert not lib.lsb_gemm_tc_pairs(M, N, K, gated)
print("ok")
"""


def test_a_plan_without_a_device():
    """(In a process of its own that is shown no device: a division by zero would end it.)"""
    done = subprocess.run([sys.executable, "-c", PROBE], capture_output=True, text=True, timeout=600,
                          env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    assert done.returncode == 0 and done.stdout.strip().endswith("ok"), (done.returncode, done.stderr[-2000:])
