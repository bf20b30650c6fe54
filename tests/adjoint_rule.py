"""The rule that picks the transposed step's tile (adjoint_rows of
csrc/step.cu), compiled for the host from its own text, so that a test can
state which tile its batch runs on."""
import os
import re
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _function(text, pattern):
    m = re.search(pattern, text, re.S | re.M)
    assert m, pattern
    return m.group(0)


def compile_rule(folder):
    """A function (mode, nx, nz, nshots, SMs) -> rows of the tile (64: 32 x 64 cells); None without a compiler."""
    gxx = shutil.which("g++")
    if gxx is None:
        return None
    text = open(os.path.join(ROOT, "seispie_b200", "csrc", "step.cu")).read()
    src = ['#include <cstdio>\n#include <cstdlib>\n#include "seispie_b200.h"\nstatic int sms;\nstatic int sm_count() { return sms; }\n',
           _function(text, r"^static int adjoint_cluster\(.*?\n\}\n"), _function(text, r"^constexpr int adjoint_ctas\(.*?\n"),
           _function(text, r"^template <int MODE>\nstatic int adjoint_rows\(.*?\n\}\n"),
           "int main(int argc, char **argv) {\n    fwi_batch b = {};\n    const int mode = atoi(argv[1]);\n"
           "    b.nx = atoi(argv[2]);\n    b.nz = atoi(argv[3]);\n    b.nshots = atoi(argv[4]);\n    sms = atoi(argv[5]);\n"
           '    printf("%d", mode == FWI_SH ? adjoint_rows<FWI_SH>(&b) : mode == FWI_PSV ? adjoint_rows<FWI_PSV>(&b) : '
           "adjoint_rows<FWI_SPIN>(&b));\n    return 0;\n}\n"]
    cpp, exe = os.path.join(folder, "rule.cpp"), os.path.join(folder, "rule")
    with open(cpp, "w") as f:
        f.write("\n".join(src))
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), cpp, "-o", exe], check=True)

    def rule(mode, nx, nz, nshots, sms=148):
        args = [str(q) for q in ({"sh": 0, "psv": 1, "spin": 2}[mode], nx, nz, nshots, sms)]
        return int(subprocess.run([exe] + args, capture_output=True, text=True, check=True).stdout)

    return rule
