"""How FP32c pencils longer than 4096 points are planned."""
import os
import subprocess

from paliwa_gb300 import build as pgbuild

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_heads_only_where_their_tensor_maps_are_accepted():
    pgbuild.build()
    out = os.path.join(pgbuild.BUILD, "long_plan_test")
    cmd = ([pgbuild.nvcc()] + pgbuild.NVCC_FLAGS +
           [os.path.join(ROOT, "tests", "cpp", "long_plan_test.cu"), "-o", out,
            "-L" + pgbuild.BUILD, "-lpaliwa_gb300", "-Xlinker",
            "-rpath=" + pgbuild.BUILD])
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([out], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
