"""The bounds-checked build takes linear offsets back to indices (kernels that walk fields
by pointers): its arithmetic on every slot of the fields' layouts, on the host."""
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_index_of_every_slot():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "index_check")
        subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                        os.path.join(ROOT, "tests", "cuda", "index_check.cu")], check=True)
        p = subprocess.run([exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout
    assert int(p.stdout) > 10000
