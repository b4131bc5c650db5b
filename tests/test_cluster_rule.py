"""Over how many CTAs K is split (csrc/cluster_rule.h), compiled for the CPU and asked about GPUs of different kinds."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sglang_b200", "csrc")
SHIM = """
#include "cluster_rule.h"
using namespace sglb200;
extern "C" void fits(const int64_t* one, const int64_t* two, int64_t sms, ClusterFits* f) {
  *f = cluster_fits_of([&](int s, int per_sm) { return per_sm == 1 ? one[s] : two[s]; }, sms);
}
extern "C" int rows(int64_t tiles, int kb, int m, const ClusterFits* f) { return rows_splits(tiles, kb, m, *f); }
extern "C" int one_launch(int64_t tiles, int kb, int most, const ClusterFits* f) { return small_splits(tiles, kb, most, *f); }
extern "C" int tile(int64_t tiles, int kb, int m, const ClusterFits* f) { return tile_splits(tiles, kb, m, *f); }
"""
ROW = ctypes.c_int64 * 17
# clusters of 0, 1, .. 16 CTAs that a B200 holds, as its driver says: one CTA on an SM, two on an SM
B200 = ([0, 148, 74, 45, 33, 26, 22, 15, 15, 15, 11, 7, 7, 7, 7, 7, 7],
        [0, 296, 148, 93, 71, 56, 45, 37, 33, 30, 26, 21, 21, 17, 14, 14, 14])
# the same where sizes above eight are refused, and where the driver says nothing
PORTABLE = tuple(r[:9] + [0] * 8 for r in B200)
SILENT = ([0] * 17, [-1] * 17)


class Fits(ctypes.Structure):
    _fields_ = [("alone", ROW), ("paired", ROW)]


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("cluster_rule")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", CSRC, "-o", str(d / "shim.so"), str(d / "shim.cpp")])
    lib = ctypes.CDLL(str(d / "shim.so"))
    lib.rows.argtypes = lib.one_launch.argtypes = lib.tile.argtypes = [ctypes.c_int64, ctypes.c_int, ctypes.c_int, ctypes.POINTER(Fits)]

    def fits(gpu):
        f = Fits()
        lib.fits(ROW(*gpu[0]), ROW(*gpu[1]), ctypes.c_int64(148), ctypes.byref(f))
        return f

    lib.of = fits
    return lib


TILES, SLABS = range(1, 300, 3), range(1, 148, 3)


def test_no_more_clusters_are_counted_than_the_driver_says(rule):
    f = rule.of(B200)
    for s in range(1, 17):
        assert 0 < f.alone[s] <= B200[0][s] and 0 < f.paired[s] <= B200[1][s], s


def test_the_one_launch_linear_takes_only_clusters_that_run_at_once(rule):
    for gpu in (B200, PORTABLE):
        f = rule.of(gpu)
        for tiles in range(1, 297):
            for kb in range(1, 129):
                s = rule.one_launch(tiles, kb, 6, f)
                assert s == 0 or tiles <= gpu[1][s], (tiles, kb, s)


@pytest.mark.parametrize("gpu", [PORTABLE, SILENT])
def test_a_size_that_the_driver_refuses_is_never_taken(rule, gpu):
    f = rule.of(gpu)
    for tiles in TILES:
        for kb in SLABS:
            for m in (17, 40, 64):
                assert 1 <= rule.rows(tiles, kb, m, f) <= 8, (tiles, kb, m)
            assert rule.one_launch(tiles, kb, 6, f) <= 8, (tiles, kb)


# (tiles, slabs, rows, CTAs measured as the faster ones): more than eight, sharing SMs, save less than they cost, but for even
# clusters with 33 to 48 rows
@pytest.mark.parametrize("tiles,kb,m,want", [(150, 126, 64, 5), (150, 126, 34, 5), (18, 91, 61, 6), (25, 77, 64, 5), (30, 34, 61, 4),
                                             (29, 35, 43, 4), (24, 80, 35, 10), (21, 96, 39, 12), (20, 107, 32, 6),
                                             (25, 78, 20, 5), (30, 64, 30, 8), (12, 127, 17, 8)])
def test_large_clusters_that_share_sms_have_to_gain_too(rule, tiles, kb, m, want):
    assert rule.rows(tiles, kb, m, rule.of(B200)) == want


def test_tiles_of_128_rows_are_split_where_that_was_faster(rule):
    """Clusters that run at once, of sizes whose exchange fits beside the operands; short K and many tiles stay whole."""
    for gpu in (B200, PORTABLE, SILENT):
        f = rule.of(gpu)
        for tiles in TILES:
            for kb in SLABS:
                s = rule.tile(tiles, kb, 128, f)
                assert s in (1, 2, 3, 4, 6, 8) and s <= kb and (s == 1 or tiles <= f.alone[s]), (tiles, kb, s)
                if kb <= 12 or tiles > 74:
                    assert s == 1
    f = rule.of(B200)
    measured = {(32, 56, 128): 4, (12, 128, 128): 8, (16, 56, 80): 6, (32, 16, 80): 4, (32, 16, 128): 1, (56, 16, 128): 1, (64, 56, 256): 2}
    assert {k: rule.tile(*k, f) for k in measured} == measured
