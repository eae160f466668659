"""Kernels chained by programmatic dependent launch read, before they wait for their predecessor, only
what no kernel writes (common.cuh chain_begin). Checked on the sources: of DevSys, whose box the volume
move's kernels write, they read the grid's shape alone, which has a memory line of its own, and nothing of DevSysD;
and they store nothing.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rainmd_b200", "csrc")
OWN_LINE = {"grid", "grid_base"}  # fields of DevSys


def early_parts():
    """(kernel, the text of each chained kernel or device function before its chain_begin())"""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*|__launch_bounds__\([^()]*\)", "", open(path).read())
        for call in re.finditer(r"chain_begin\(\)", text):
            head = [m for m in re.finditer(r"(?:__global__|__device__)[^;{}]*?(\w+)\(([^;{}]*)\)\s*\{",
                                           text[:call.start()])][-1]
            out.append((f"{os.path.basename(path)}:{head.group(1)}", text[head.end():call.start()]))
    return out


EARLY = early_parts()


def test_every_chained_kernel_is_found():
    names = {n.split(":")[1] for n, _ in EARLY}
    assert {"k_spread", "k_fft_r2c", "k_fft_c2r", "k_fft_planes", "k_gather4", "process_unit"} <= names


@pytest.mark.parametrize("name,before", EARLY, ids=[f"{n}-{k}" for k, (n, _) in enumerate(EARLY)])
def test_reads_before_the_wait(name, before):
    assert not re.search(r"\bsysd\b", before)
    for ref in re.findall(r"DevSys\s*&\s*(\w+)\s*=", before):
        assert set(re.findall(rf"\b{ref}\.(\w+)", before)) <= OWN_LINE, name
    # otherwise DevSys is not touched
    assert not re.search(r"\bsys\s*\[", re.sub(r"DevSys\s*&\s*\w+\s*=\s*sys\[", "", before)), name
    stores = re.findall(r"\b(posq|vel|force|half|real_grid|fixed_grid|spos|e_pme|e_pme_vir|disp|diag)\s*\[[^\]]*\]\s*=",
                        before)
    assert not stores, (name, stores)


def test_fields_read_early_have_a_line_of_their_own():
    struct = re.search(r"struct DevSys \{(.*?)\n\};", open(os.path.join(CSRC, "common.cuh")).read(), re.S).group(1)
    struct = re.sub(r"//[^\n]*", "", struct)
    line = re.search(r"alignas\(128\)(.*?)alignas\(128\)", struct, re.S)
    assert line, "no memory line set apart"
    assert set(re.findall(r"(\w+)(?:\[\d+\])?\s*;", line.group(1))) == OWN_LINE
