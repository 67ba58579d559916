"""How the full-sum solver's rows are cut into units (rows_plan.h), checked on
the host."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run_program(tmp_path, body):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src = tmp_path / "plan.cu"
    src.write_text('#include "rows_plan.h"\n#include <algorithm>\n#include <cstdio>\nusing namespace ccf;\n'
                   "int main()\n{\n    int bad = 0;\n" + body + '    std::printf("bad %d\\n", bad);\n    return bad != 0;\n}\n')
    exe = tmp_path / "plan"
    r = subprocess.run([nvcc, "-std=c++20", "-I", os.path.join(ROOT, "ccf_gb300", "csrc"), "-I",
                        os.path.join(ROOT, "include"), str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert out.stdout.strip().endswith("bad 0")


def test_a_ticket_holds_any_number_of_units(tmp_path):
    """The units of a sums phase in a row's ticket, from one star to millions,
    and drawn to the last one."""
    run_program(tmp_path, r"""
    for (long long n : {1LL, 2000LL, 20000LL, 604000LL, 605000LL, 606000LL, 610000LL, 1000000LL, 3000000LL})
    {
        const int R = (int)(2 * n), N = (int)n, nch = (R + CHUNK - 1) / CHUNK + (N + CHUNK - 1) / CHUNK;
        for (int total : {1, R / 1000 + 1, R})
        {
            const SumsShape p = sums_shape(total, source_split(total, 16), R, N, nch, 1, 152);
            const int units = p.tiles * p.groups;
            if (units < 1 || p.groups * p.chunks < nch) bad++;
            unsigned long long t = ticket_open(units) | 1ull;
            if (ticket_units(t) != units || ticket_next(t) != 1) bad++;
            t += (unsigned long long)units - 1;   /* every unit drawn, and more CTAs asking */
            if (ticket_units(t) != units || ticket_next(t) != units) bad++;
            t += 304;
            if (ticket_units(t) != units || ticket_next(t) != units + 304) bad++;
        }
    }
""")
