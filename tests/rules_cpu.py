"""csrc/am_rules.h compiled for the host: a shim's functions, through ctypes."""
import ctypes as C
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def rules(tmp_path, body):
    """Compiles `body` (extern "C" functions that may use namespace am) and loads it."""
    src, so = tmp_path / "shim.cpp", tmp_path / "shim.so"
    src.write_text('#include "am_rules.h"\nusing namespace am;\nextern "C" {\n%s\n}\n' % body)
    inc = os.path.join(ROOT, "analyticmesh_gb300", "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", inc, "-o", str(so), str(src)], check=True)
    return C.CDLL(str(so))
