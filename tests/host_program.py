"""Programs of tests/host linked with the library's objects and a CUDA runtime without a device
(tests/host/runtime.cpp): for what the host side does when an allocation is refused."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HOST = os.path.join(ROOT, "tests", "host")


def compile_and_run(name, tmp_path, *args):
    """Compiles tests/host/<name>.cpp and runs it; its output. Fails on a non-zero exit."""
    import build  # sitk-rs_b200/build.py
    build.build()
    objects = [os.path.join(build.BUILD, s + ".o") for s in build.CU_SOURCES + build.CPP_SOURCES]
    inc = ["-I", build.INCLUDE, "-I", build.CSRC, "-I", HOST, "-I", "/usr/local/cuda/include"]
    own = []
    for src in (name, "runtime"):
        o = str(tmp_path / (src + ".o"))
        subprocess.run(["g++", "-std=c++17", "-O1", "-g", *inc, "-c", os.path.join(HOST, src + ".cpp"), "-o", o], check=True)
        own.append(o)

    def symbols(flag, files):
        out = subprocess.run(["nm", flag, *files], capture_output=True, text=True, check=True).stdout
        return set(re.findall(r"\b(_{0,2}cuda\w+)$", out, re.M))

    rest = symbols("-u", objects + own) - symbols("--defined-only", own + objects)
    stubs = tmp_path / "stubs.c"
    stubs.write_text("".join(f"long {s}() {{ return 0; }}\n" for s in sorted(rest)))
    subprocess.run(["gcc", "-c", str(stubs), "-o", str(tmp_path / "stubs.o")], check=True)
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-o", exe, *own, str(tmp_path / "stubs.o"), *objects, "-lz", "-lpthread", "-ldl"], check=True)
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
