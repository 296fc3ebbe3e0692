"""Tables of the band-wise dedispersion kernel, walked on the host.

A small C++ program (band_tables_check.cpp) builds the kernel's tables for a
delay table and repeats the kernel's index arithmetic -- tiles, staged rows,
windows, patterns, skewed accumulators, output ranges -- on whole numbers, so
the result must equal the plain sum exactly and every access must lie inside
its tile row."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("band") / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "vlite-frb_b200", "csrc"),
                    os.path.join(ROOT, "tests", "band_tables_check.cpp"), "-o", exe], check=True)

    def run(off, nt, row0=0, nvalid=None, tt=9, over=0):
        off = np.asarray(off, np.int64)
        nvalid = nt + int(off.max()) if nvalid is None else nvalid
        text = f"{off.shape[0]} {off.shape[1]} {row0} 0 {nvalid} {nt} {tt} {over}\n"
        text += " ".join(map(str, off.ravel()))
        r = subprocess.run([exe], input=text, capture_output=True, text=True)
        assert r.returncode in (0, 3), r.stdout
        return r.returncode == 0, r.stdout

    return run


def _table(O, ndm, dm_max, nch=96, chanbw=0.5, tchan=1e-3, dm_min=0.0):
    dms = np.linspace(dm_min, dm_max, ndm).astype(np.float32)
    return O.delay_table(dms, 384.0, chanbw, tchan, nch)[0]


# samples per lane and elements read past a window: FP32, FP16 (a word), int8 (a word)
FORMS = [(9, 0), (10, 2), (8, 4)]


@pytest.mark.parametrize("tt,over", FORMS)
@pytest.mark.parametrize("ndm,dm_max,nt,row0", [
    (8, 3.0, 1, 0), (9, 0.5, 479, 3), (49, 40.0, 481, 16), (48, 10.0, 960, 500), (332, 20.0, 290, 9), (650, 60.0, 100, 5), (61, 200.0, 700, 1000003),
    (100, 30.0, 33, 7)])
def test_tables_give_the_plain_sum(check, O, ndm, dm_max, nt, row0, tt, over):
    ok, text = check(_table(O, ndm, dm_max), nt, row0=row0, tt=tt, over=over)
    assert ok, "the kernel applies to every equally spaced list of eight trials or more"
    print(text)


def test_tables_with_more_valid_rows_and_an_offset_list(check, O):
    ok, _ = check(_table(O, 24, 90.0, dm_min=60.0), 500, row0=77, nvalid=4000)
    assert ok


def test_shifts_off_the_staircase_take_the_generic_path(check, O):
    off = _table(O, 64, 20.0)
    off[17:19, 40] += 1  # two delays off the staircase, in one channel: under 5% of the pairs
    ok, text = check(off, 200)
    assert ok and "generic 1" in text


def test_refused_tables(check, O):
    rng = np.random.default_rng(1)
    assert not check(_table(O, 7, 3.0), 50)[0]  # fewer than a group
    uneven = np.sort(rng.uniform(0, 200, 40)).astype(np.float32)
    assert not check(O.delay_table(uneven, 384.0, 0.5, 1e-3, 96)[0], 50)[0]
    falling = _table(O, 16, 40.0)[::-1]
    assert not check(falling, 50)[0]
