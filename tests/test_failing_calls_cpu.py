"""Every call that the attention layer makes into the CUDA layer fails once, on the CPU: tests/failing_calls_check.c."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_failing_call_leaves_a_block_behind(tmp_path):
    exe, src = tmp_path / "failing_calls_check", os.path.join(ROOT, "boat_b200", "csrc")
    subprocess.run(["gcc", "-std=c11", "-O1", "-g", "-D_GNU_SOURCE", "-fsanitize=address,undefined", "-fno-sanitize-recover=all",
                    "-I" + os.path.join(ROOT, "include"), "-o", str(exe), os.path.join(ROOT, "tests", "failing_calls_check.c")] +
                   [os.path.join(src, f) for f in ("layers/attention.c", "core/stage.c", "core/memory.c", "core/tensor.c")] + ["-lm"],
                   check=True)
    env = {k: v for k, v in os.environ.items() if not k.startswith("BOAT_")}
    env["ASAN_OPTIONS"] = "detect_leaks=0"
    proc = subprocess.run([str(exe)], env=env, stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True, timeout=300)
    assert proc.returncode == 0 and proc.stdout.endswith("ok\n"), proc.stdout[-2000:]
