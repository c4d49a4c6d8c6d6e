"""Rules and index arithmetic that host and device code share, compiled for the host."""
import os
import subprocess

import pytest

from tensilelite_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def host_program(tmp_path, body):
    """Output lines of a C++ program with the library's internal header."""
    include = os.path.join(os.path.dirname(os.path.dirname(_build.nvcc())), "include")
    src = ('#include <cstdio>\n#include <cstring>\n#include <vector>\n#include "tensilelite_gb300/csrc/tl_internal.h"\n'
           "using namespace tl;\nint main()\n{\n" + body + "\n    return 0;\n}\n")
    exe = str(tmp_path / "probe")
    r = subprocess.run(["g++", "-std=c++17", "-x", "c++", "-I", ROOT, "-I", include, "-o", exe, "-"], input=src, text=True,
                       capture_output=True)
    assert r.returncode == 0, r.stderr
    return subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()


@pytest.mark.parametrize("units,workers,beside_others,mode", [(64, 152, 0, 1), (64, 152, 1, 2), (152, 152, 1, 2),
                                                             (153, 152, 0, 0), (153, 152, 1, 0), (0, 152, 0, 0)])
def test_splits_rely_on_each_other_only_alone(tmp_path, units, workers, beside_others, mode):
    out = host_program(tmp_path, f'    printf("%d", tc_par_reduce({units}, 0, {workers}, {beside_others}));')
    assert out == [str(mode)]
