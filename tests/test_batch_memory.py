"""Device memory of the batched solver's slices (csrc/batch.cu), checked on the CPU
through a host-only helper (tests/batch_memory.cu) on a device of a given size: what
needs memory later takes the slices', and a refused call leaves nothing half made."""

import os
import subprocess

import sovereign_solver_gb300._build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def test_slices_give_way(tmp_path):
    exe = str(tmp_path / "batch_memory")
    cmd = [B.nvcc(), "-gencode", "arch=compute_103a,code=compute_103a", "-Xcicc", "-O0", "-O0", "-std=c++17",
           f"-I{B.CSRC}", f"-I{B.INCLUDE}", os.path.join(HERE, "batch_memory.cu"), "-o", exe, "-lcudart_static", "-lrt",
           "-lpthread", "-ldl"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")                # its launches must find no device
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60, env=env)
    assert r.returncode == 0 and "FAILED" not in r.stdout, r.stdout + r.stderr
