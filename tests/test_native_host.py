"""Host logic of the CUDA sources, compiled with stand-ins for the CUDA calls
it makes: no GPU needed."""
import os
import subprocess

from libspimage_b200 import build as b

HERE = os.path.dirname(os.path.abspath(__file__))


def run_native(tmp_path, name, *flags):
    exe = str(tmp_path / name)
    cmd = [b._nvcc(), *b.ARCH, "-std=c++17", "-I", b.INCLUDE, "-I", b.CSRC, "-o", exe,
           os.path.join(HERE, "native", name + ".cu"), *flags]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_shared_memory_limit_never_falls(tmp_path):
    """Contexts of different line lengths on different host threads."""
    run_native(tmp_path, "smem_limit")


def test_transform_tables_are_up_before_the_first_pass(tmp_path):
    """A one-shot context's tables are not left on their way on another stream."""
    lib = b.build()
    fast = ["-O0", "-Xcicc", "-O0", "-Xptxas", "-O0", "-diag-suppress", "177"]  # nothing here runs on a device
    run_native(tmp_path, "table_upload", *fast, lib, "-Xlinker", "-rpath=" + os.path.dirname(lib))
