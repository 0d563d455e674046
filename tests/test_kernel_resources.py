"""The hot kernels compile for sm_100a without local memory: no stack frame
and no register spills.  A value that falls to local memory costs these
loops several percent (a float4 taken by reference in the kick's buffer
tail cost 6 % of the kick), so the property is checked on the CPU with
nvcc -Xptxas -v, with the library's own build flags.  The kernels around them
may spill no more than they do (the register bound that makes them spill was
measured faster than the next lower occupancy)."""
import concurrent.futures
import os
import re
import subprocess
import tempfile

import pytest

from tigerpm_b200 import build as B

# source file -> kernels (a regex on the mangled name) that must use neither
# a stack frame nor spills
HOT = {
    "kick_pme.cu": [r"k_kick_pme", r"k_kick_batch", r"k_kick_slots"],
    "gravity_long.cu": [r"k_deposit"],
    "fft3d.cu": [r"k_line_x_greenILi768E", r"k_line_z_r2cILi768E"],
}

# source file -> kernels and the bytes of spill stores or loads they may have
# (the interpolation's stack frame holds its weights, which are indexed)
SPILLS = {
    "kick_pme.cu": {r"k_interp_direct": 4, r"k_interp_items": 16, r"k_interp_slots": 80, r"k_interp_tile": 0, r"k_item_": 0},
    "chainmesh.cu": {r"k_finish": 24, r"k_level_": 0, r"k_gather": 0, r"k_records": 0, r"k_scan_": 0},
    "fft3d.cu": {r"k_line_x_green": 0, r"k_line_y": 0, r"k_line_z_r2c": 0, r"k_line_z_c2r": 24},
}


def ptxas_report(src):
    """{mangled kernel name: (stack bytes, spill store bytes, spill load bytes)}"""
    with tempfile.TemporaryDirectory() as d:
        cmd = [B.nvcc()] + B.ARCH + B.NVCC_FLAGS + ["-Xptxas", "-v", "-c", os.path.join(B.CSRC, src),
                                                   "-o", os.path.join(d, "x.o")]
        out = subprocess.run(cmd, capture_output=True, text=True, check=True).stderr
    report, name = {}, None
    for line in out.splitlines():
        m = re.search(r"Compiling entry function '([^']+)'", line)
        if m:
            name = m.group(1)
            continue
        m = re.search(r"(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", line)
        if m and name:
            report[name] = tuple(int(g) for g in m.groups())
            name = None
    return report


def nvcc_available():
    try:
        B.nvcc()
        return True
    except RuntimeError:
        return False


@pytest.fixture(scope="module")
def reports():
    if not nvcc_available():
        pytest.skip("nvcc not found")
    files = sorted(set(HOT) | set(SPILLS))
    with concurrent.futures.ThreadPoolExecutor(len(files)) as ex:
        return dict(zip(files, ex.map(ptxas_report, files)))


def test_hot_kernels_use_no_local_memory(reports):
    for src, patterns in HOT.items():
        for pat in patterns:
            hits = {k: v for k, v in reports[src].items() if re.search(pat, k)}
            assert hits, (src, pat)
            bad = {k: v for k, v in hits.items() if any(v)}
            assert not bad, (src, pat, bad)


def test_other_kernels_spill_no_more_than_they_do(reports):
    for src, patterns in SPILLS.items():
        for pat, most in patterns.items():
            hits = {k: v for k, v in reports[src].items() if re.search(pat, k)}
            assert hits, (src, pat)
            bad = {k: v for k, v in hits.items() if max(v[1:]) > most}
            assert not bad, (src, pat, bad)
