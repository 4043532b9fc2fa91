"""populate_host (host mesh arrays' pages before the device writes there)."""
import os
import subprocess

from tests.test_cpp_reconstructor import BUILD, ROOT


def test_first_refusal_ends_it():
    from fluidsurfacereconstructiongpu_gb300 import build as B
    os.makedirs(BUILD, exist_ok=True)
    lib_dir = os.path.dirname(B.LIB_PATH)
    exe = os.path.join(BUILD, "populate")
    subprocess.run(["g++", "-std=c++17", "-O1", "-rdynamic", os.path.join(ROOT, "tests", "cpp", "populate.cpp"),
                    "-o", exe, "-L", lib_dir, "-lfsr_gb300", f"-Wl,-rpath,{lib_dir}"], check=True)
    assert subprocess.run([exe], check=True, stdout=subprocess.PIPE, text=True).stdout == "ok\n"
