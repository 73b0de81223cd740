"""When MD runs follow the host's list schedule (csrc/nb_foresight.h), compiled as host code: runs left to the
device after lists were outrun, more of them each time, fewer again after runs that kept their schedule."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "moil_fnrfd_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include "nb_foresight.h"
int main(int argc, char **argv)
{
    // o: a foreseen run outruns its lists, k: it keeps them, r: a new system; between them, runs on the device
    ListForesight f;
    for (const char *c = argv[1]; *c; ++c) {
        int device = 0;
        while (!f.host(true)) { f.begin(); ++device; }
        printf("%d ", device);
        f.begin();
        if (*c == 'o') f.outrun();
        else if (*c == 'k') f.kept();
        else f.reset();
    }
    printf("%d\n", f.host(false) ? 1 : 0);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cc = shutil.which("g++") or shutil.which("nvcc")
    if cc is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("foresight")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run([cc, "-O1", "-I", CSRC, str(d / "main.cpp"), "-o", str(d / "run")], check=True)
    return str(d / "run")


@pytest.mark.parametrize("events,device_runs", [
    ("kkk", [0, 0, 0]),
    ("ooooooook", [0, 2, 6, 14, 30, 62, 64, 64, 64]),
    ("ooookkkkoo", [0, 2, 6, 14, 30, 0, 0, 0, 0, 4]),       # 30 halved four times leaves 1, the next is 4
    ("oooorok", [0, 2, 6, 14, 30, 0, 2]),                   # a new system forgets
])
def test_runs_left_to_the_device(program, events, device_runs):
    out = [int(x) for x in subprocess.run([program, events], check=True, capture_output=True, text=True).stdout.split()]
    assert out[:-1] == device_runs and out[-1] == 0        # and never without a period
