"""Which kernel launches may run beside the ones before them (csrc/cuda/launch_order.h, which makes no CUDA call), compiled for
the CPU: tests/launch_order_check.cpp."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launch_order(tmp_path):
    exe = tmp_path / "launch_order_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-Wall", "-Wextra", "-Werror", "-fsanitize=address,undefined",
                    "-fno-sanitize-recover=all", "-I" + os.path.join(ROOT, "boat_b200", "csrc", "cuda"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "launch_order_check.cpp")], check=True)
    env = dict(os.environ, ASAN_OPTIONS="detect_leaks=0")
    proc = subprocess.run([str(exe)], env=env, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert proc.returncode == 0 and proc.stdout.endswith("ok\n"), proc.stdout[-2000:]


def test_what_others_put_on_the_stream_is_announced(tmp_path):
    """NCCL's collectives and the self test's kernel: tests/foreign_launches_check.cpp."""
    exe, nccl, src = tmp_path / "foreign_launches_check", tmp_path / "libplayed_nccl.so", os.path.join(ROOT, "boat_b200", "csrc", "cuda")
    nvcc = ["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + os.path.join(ROOT, "include"), "-I" + src,
            os.path.join(ROOT, "tests", "foreign_launches_check.cpp")]
    subprocess.run(nvcc + ["-DPLAYED_NCCL", "-shared", "-Xcompiler", "-fPIC", "-o", str(nccl)], check=True)
    subprocess.run(nvcc + [os.path.join(src, "comm.cu"), os.path.join(src, "selftest.cu"), "-o", str(exe), "-ldl"], check=True)
    proc = subprocess.run([str(exe)], env=dict(os.environ, BOAT_NCCL_LIB=str(nccl)), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True,
                          timeout=300)
    assert proc.returncode == 0 and proc.stdout.endswith("ok\n"), proc.stdout[-2000:]
