"""Small C++ programs against the engine's library, for what its C interface does not reach."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
PKG = ROOT / "simulador_quantico_b200"
CUDA = Path("/usr/local/cuda")


def run(tmp_path, source, *args):
    """Compiles `source` (with the engine's internal header at hand), runs it and returns its output."""
    src, exe = tmp_path / "prog.cpp", tmp_path / "prog"
    src.write_text('#include <cuda_runtime.h>\n#include <cstdio>\n#include <cstdlib>\n#include "hgm_internal.h"\n'
                   "using namespace hgm;\n" + source)
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{ROOT / 'include'}", f"-I{PKG / 'csrc'}", f"-I{CUDA / 'include'}",
                    src, "-o", exe, f"-L{PKG / 'lib'}", "-lhgm_b200", f"-Wl,-rpath,{PKG / 'lib'}",
                    f"-L{CUDA / 'lib64'}", "-lcudart_static", "-ldl", "-lrt", "-lpthread"], check=True)
    return subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True, timeout=300).stdout
