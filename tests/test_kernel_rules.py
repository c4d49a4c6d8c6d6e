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


@pytest.mark.parametrize("odd", [0, 1])
def test_eight_halves_read_nothing_else(tmp_path, odd):
    """Elements 1 .. 8 of a guarded buffer: the values in order, and no read outside [0, 8)."""
    body = f"""
    uint16_t src[8];
    for (int i = 0; i < 8; ++i) src[i] = static_cast<uint16_t>(0x1100 * (i + 1) + i);
    int low = 100, high = -100;
    const auto seen = [&](int a, int b) {{ if (a < low) low = a; if (b > high) high = b; }};
    uint32_t v[4];
    load_eight16({odd}, [&](int e) {{ seen(e, e); return static_cast<uint32_t>(src[e & 7]); }},
                 [&](int e) {{ seen(e, e + 1); return src[e & 7] | (static_cast<uint32_t>(src[(e + 1) & 7]) << 16); }}, v);
    int bad = 0;
    for (int i = 0; i < 8; ++i) bad += (v[i / 2] >> (16 * (i & 1)) & 0xffff) != src[i];
    printf("%d %d %d", low, high, bad);"""
    assert host_program(tmp_path, body) == ["0", "7", "0"]
