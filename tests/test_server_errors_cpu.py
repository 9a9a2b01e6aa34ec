"""The server's error paths from many threads on the CPU: statuses and
messages stay each call's own (tests/server_errors_check.cu), once as built
and, where the compiler's thread sanitizer runs, once under it."""
import glob
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("sanitize", [False, True])
def test_server_errors_from_many_threads(tmp_path, sanitize):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    objs = [o for o in glob.glob(os.path.join(ROOT, "rtscan_b200", "_build", "*.o")) if not o.endswith("serve.cpp.o")]
    if not os.path.exists(nvcc) or not objs:
        pytest.skip("needs nvcc and the library's objects (run the build first)")
    flags = ["-Xcompiler", "-fsanitize=thread,-g"] if sanitize else []
    if sanitize:  # does a program run under it here?
        src, probe = tmp_path / "probe.cu", tmp_path / "probe"
        src.write_text("int main() { return 0; }\n")
        built = subprocess.run([nvcc, *flags, str(src), "-o", str(probe)], capture_output=True, timeout=300)
        if built.returncode or subprocess.run([str(probe)], capture_output=True, timeout=60).returncode:
            pytest.skip("no thread sanitizer here")
    out = str(tmp_path / "server_errors_check")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                        "-I", os.path.join(ROOT, "include"), *flags,
                        os.path.join(ROOT, "tests", "server_errors_check.cu"), *objs,
                        "-Xlinker", "--as-needed", "-lcuda", "-o", out], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([out, "500" if sanitize else "20000"], capture_output=True, text=True, timeout=600,
                       env={**os.environ, "TSAN_OPTIONS": "halt_on_error=1 exitcode=66"})
    assert r.returncode == 0 and "server errors ok" in r.stdout, (r.returncode, r.stderr[-3000:])
