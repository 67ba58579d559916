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
            const SumsShape p = sums_shape(total, source_split(total, 16), R, N, nch, 1, 152, false);
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


def test_a_rows_partial_sums_stay_within_their_memory(tmp_path):
    """Every sweep of a row fits the bytes its plan gives it, whole sums or one
    per chunk, and from 52 000 stars on those bytes grow with the stars and no
    longer with their square."""
    run_program(tmp_path, r"""
    for (long long n : {1LL, 31LL, 700LL, 5000LL, 20000LL, 52000LL, 60000LL, 100000LL, 605000LL, 2000000LL})
        for (int cluster : {1, 2, 4, 8, 16})
            for (bool mixed : {false, true})
                for (long long limit : {1LL, 100000LL, ROWS_PART_BYTES})
                {
                    const int R = (int)(2 * n), N = (int)n, nch = (R + CHUNK - 1) / CHUNK + (N + CHUNK - 1) / CHUNK;
                    const long long bytes = row_part_bytes(R, N, cluster, mixed, limit);
                    if (bytes % 16 != 0) bad++;
                    if (limit == ROWS_PART_BYTES && bytes > std::max(ROWS_PART_BYTES, 64LL * R + 32LL * 21 * TILE * 8)) bad++;
                    for (int total = 1; total <= R; total += total < 20000 ? 1 : 997)
                    {
                        const int S = source_split(total, cluster);
                        const bool whole = sums_whole(total, S, nch, mixed, limit);
                        const long long need = (long long)S * total * (whole ? 2 * 16 : nch * (mixed ? 8 : 16));
                        if (need > bytes) bad++;
                        const SumsShape p = sums_shape(total, S, R, N, nch, 1, 152, whole);
                        if (whole && p.groups != 1) bad++;
                    }
                    for (long long rows : {1LL, 64LL, 12288LL})
                    {
                        const RowsScratch q = rows_scratch(bytes, R, rows);
                        if (q.slots < 1 || q.slots > rows || (q.slots > 1 && q.bytes() > ROWS_PART_BYTES)) bad++;
                    }
                }
""")
