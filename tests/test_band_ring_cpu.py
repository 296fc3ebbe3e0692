"""Staging of the band-wise dedispersion kernel on tight rings, walked on the host.

A ring need only hold the valid rows.  band_ring_check.cpp repeats the kernel's
staging arithmetic for rings of the smallest sizes that a call may use, row0
anywhere on them, for the 16-byte groups of each storage form."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("ring") / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "vlite-frb_b200", "csrc"),
                    os.path.join(ROOT, "tests", "band_ring_check.cpp"), "-o", exe], check=True)

    def run(off, nt, row0, ring, nvalid, tt, vec):
        text = f"{off.shape[0]} {off.shape[1]} {row0} {ring} {nvalid} {nt} {tt} {vec}\n"
        r = subprocess.run([exe], input=text + " ".join(map(str, off.ravel())), capture_output=True, text=True)
        assert r.returncode == 0, r.stdout

    return run


# samples per lane and rows of 16 bytes: FP32, FP16, int8
@pytest.mark.parametrize("tt,vec", [(9, 4), (10, 8), (8, 16)])
@pytest.mark.parametrize("ndm,dm_max,nt", [(17, 1.0, 1), (17, 2.6, 1), (17, 20.0, 7), (40, 30.0, 300), (60, 4.0, 97),
                                           (400, 60.0, 20)])
def test_copies_stay_inside_the_smallest_ring(check, O, ndm, dm_max, nt, tt, vec):
    dms = np.linspace(0, dm_max, ndm).astype(np.float32)
    off, _ = O.delay_table(dms, 384.0, 1.0, 1e-3, 64)
    need = nt + int(off.max())
    ring = max(vec, 1 << (need - 1).bit_length())
    rng = np.random.default_rng(ndm + nt)
    for nvalid in (need, ring):
        for row0 in [0, 1, ring - 1, 71, 1039] + [int(x) for x in rng.integers(0, 8 * ring, 4)]:
            check(off, nt, row0, ring, nvalid, tt, vec)
