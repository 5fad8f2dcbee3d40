"""Decode attention's split of its heads, as the host works it out, over many sizes and numbers of SMs (CPU only)."""
import glob
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_split_of_the_heads_is_resident(tmp_path):
    import __graft_entry__ as g
    g.build()
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = str(tmp_path / "check")
    pkg = os.path.join(ROOT, "ml-drift_b200")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-Wall", "-o", exe, os.path.join(ROOT, "tests", "attn_shape_check.cc"),
                           *sorted(glob.glob(os.path.join(pkg, "build", "*.o"))), "-I", os.path.join(ROOT, "include"), "-I",
                           os.path.join(pkg, "csrc"), "-I", os.path.join(cuda, "include"), "-L", os.path.join(cuda, "lib64"),
                           "-lcudart", "-ldl", "-Wl,-rpath," + os.path.join(cuda, "lib64")])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and "shapes" in out.stdout, out.stdout
