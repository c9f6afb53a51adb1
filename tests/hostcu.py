"""Compiles a host program against the engine's internal headers and runs it
(no GPU): the index arithmetic that kernels and host code share."""
import subprocess

from fsig_gb300 import _build


def run(tmp_path, body: str) -> None:
    """`body` is the inside of main(); check(ok, line) counts failures."""
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text('#include <cstdio>\n#include <cstdlib>\n#include <sys/mman.h>\n#include "common.cuh"\n#include "queue.cuh"\n'
                   "static int bad = 0;\n"
                   "static void check(bool ok, int line) { if (!ok) { bad++; std::printf(\"line %d\\n\", line); } }\n"
                   "#define CHECK(x) check((x), __LINE__)\nusing namespace fsig;\n"
                   "int main() {\n#line 1\n" + body + "\n  return bad ? 1 : 0;\n}\n")
    subprocess.run([_build._nvcc(), *_build.ARCH, "-std=c++17", "-O1", "--expt-relaxed-constexpr",
                    "-I", str(_build.CSRC), "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
