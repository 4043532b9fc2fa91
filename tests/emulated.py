"""Builds and runs a test program around the library's kernel sources on the
host (tests/cpp/warp_emul.h): the sources are copied to tests/_build with what a
host compiler does not take replaced (the two approximate reciprocals, the
dynamic shared array's qualifier)."""
import atexit
import functools
import os
import pathlib
import re
import shutil
import subprocess

ROOT = pathlib.Path(__file__).resolve().parents[1]
CSRC = ROOT / "fluidsurfacereconstructiongpu_gb300" / "csrc"
BUILD = ROOT / "tests" / "_build" / "emulated"


def _sources():
    out = BUILD / "pkg" / "csrc"
    out.mkdir(parents=True, exist_ok=True)
    shutil.copytree(ROOT / "include", BUILD / "include", dirs_exist_ok=True)
    for path in CSRC.iterdir():
        if path.suffix not in (".cu", ".cuh", ".h"):
            continue
        text = path.read_text().replace("extern __shared__", "extern")
        text = re.sub(r'asm\("rsqrt\.approx.*', "y = 1.0f / std::sqrt(x);", text)
        text = re.sub(r'asm\("rcp\.approx.*', "y = 1.0f / d;", text)
        (out / path.name).write_text(text)
    return out


@functools.lru_cache(maxsize=None)
def build(program):
    out = BUILD / f"{program}.{os.getpid()}"
    csrc = _sources()
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    # (host code of other source files is not called)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-ffp-contract=off", f"-I{csrc}", f"-I{cuda}",
                    str(ROOT / "tests" / "cpp" / f"{program}.cpp"), "-o", str(out),
                    "-Wl,--unresolved-symbols=ignore-all"], check=True)
    atexit.register(lambda: out.unlink(missing_ok=True))
    return out


def run(program, *args, timeout=300):
    """Compiles tests/cpp/<program>.cpp and returns what it prints."""
    return subprocess.run([str(build(program)), *map(str, args)], check=True, timeout=timeout, stdout=subprocess.PIPE,
                          text=True).stdout
