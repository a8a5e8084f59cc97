"""The launch rules (kpt_rules.h) on the host, against times measured on the
GB300 (152 SMs) at sizes, substeps and populations on both sides of each line:
what a rule picks may not be slower than the simple choice it departs from."""
from __future__ import annotations

import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "kokkos-particletransport_gb300", "csrc")
SMS = 152
SHIM = """
#include "kpt_rules.h"
extern "C" int records_pay(int focused, int learned, uint64_t particles, uint64_t points,
                           double dt_min, double dt_max, int sms) {
    return kpt::records_pay({focused != 0, learned != 0, particles, points, dt_min, dt_max, sms});
}
extern "C" int batch_records_pay(int focused, int fixed, int runs, double particles, double points,
                                 double steps, int sms) {
    return kpt::batch_records_pay({focused != 0, false, fixed != 0, (size_t)runs, particles, points,
                                   steps, sms});
}
extern "C" int batch_point_threads(uint64_t particles, int fixed, int fit, int sms) {
    return kpt::batch_point_threads(particles, fixed != 0, fit, sms);
}
extern "C" int point_blocks(uint64_t particles, int fixed, double table_bytes, double l2_bytes,
                            int sms) {
    return kpt::point_blocks(particles, fixed != 0, table_bytes, l2_bytes, sms);
}
extern "C" int f64_blocks_per_sm(uint64_t particles, int fixed, uint64_t lanes, int most,
                                 int requested) {
    return kpt::f64_blocks_per_sm(particles, fixed != 0, lanes, most, requested);
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    path = tmp_path_factory.mktemp("rules")
    src, so = str(path / "rules.cpp"), str(path / "rules.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", CSRC, src, "-o", so],
                   check=True)
    lib = ctypes.CDLL(so)
    u64, dbl, i32 = ctypes.c_uint64, ctypes.c_double, ctypes.c_int
    lib.records_pay.argtypes = [i32, i32, u64, u64, dbl, dbl, i32]
    lib.batch_records_pay.argtypes = [i32, i32, i32, dbl, dbl, dbl, i32]
    lib.batch_point_threads.argtypes = [u64, i32, i32, i32]
    lib.point_blocks.argtypes = [u64, i32, dbl, dbl, i32]
    lib.f64_blocks_per_sm.argtypes = [u64, i32, u64, i32, i32]
    return lib


# focused, nx, ny, particles, substeps, and ms of an interval whose tables are
# new: on the point tables, on records (plain closures, fixed steps)
SINGLE = [
    (0, 1024, 1024, 126814, 100, 0.785, 0.958), (0, 1024, 1024, 126814, 200, 1.484, 1.580),
    (0, 1024, 1024, 211356, 100, 1.110, 1.221), (0, 1024, 1024, 211356, 400, 4.297, 3.710),
    (0, 1024, 1024, 253628, 50, 0.712, 0.770), (0, 1024, 1024, 253628, 200, 2.667, 2.242),
    (0, 1024, 2048, 126567, 200, 1.521, 1.992), (0, 1024, 2048, 126567, 400, 2.955, 3.276),
    (0, 1024, 2048, 253134, 100, 1.372, 1.706), (0, 1024, 2048, 253134, 200, 2.679, 2.839),
    (0, 1024, 2048, 421891, 100, 2.193, 2.332), (0, 1024, 2048, 421891, 400, 8.641, 7.137),
    (0, 1024, 2048, 506269, 50, 1.320, 1.540), (0, 1024, 2048, 506269, 400, 10.230, 8.161),
    (0, 2048, 4096, 252396, 400, 6.520, 7.684), (0, 2048, 4096, 504792, 200, 5.529, 7.922),
    (0, 2048, 4096, 504792, 400, 10.483, 13.901), (0, 2048, 4096, 1009584, 100, 5.125, 7.253),
    (0, 2048, 4096, 1009584, 400, 19.979, 22.901), (0, 2048, 4096, 1682640, 100, 8.344, 9.967),
    (0, 2048, 4096, 2019168, 50, 5.112, 6.470), (0, 2048, 4096, 2019168, 100, 9.970, 11.107),
    (0, 512, 1024, 124655, 50, 0.409, 0.437), (0, 512, 1024, 124655, 200, 1.458, 1.211),
    (0, 1500, 1500, 226201, 400, 4.692, 5.077), (0, 1500, 1500, 361922, 400, 7.483, 6.580),
    (0, 256, 4096, 170560, 100, 0.916, 0.973), (0, 256, 4096, 170560, 400, 3.543, 2.822),
    (1, 512, 1024, 124655, 50, 0.608, 0.647), (1, 512, 1024, 132081, 400, 4.516, 3.724),
    (1, 700, 800, 140937, 100, 1.195, 1.199), (1, 700, 800, 140937, 400, 4.698, 3.942),
    (1, 1500, 1500, 226201, 400, 7.120, 7.884), (1, 1500, 1500, 531573, 400, 16.307, 14.097),
    (1, 256, 4096, 213200, 100, 1.697, 1.884), (1, 256, 4096, 265434, 400, 8.209, 6.202),
    (1, 1024, 1024, 126814, 100, 1.215, 1.414), (1, 1024, 1024, 126814, 200, 2.299, 2.526),
    (1, 1024, 1024, 211356, 100, 1.688, 1.903), (1, 1024, 1024, 211356, 200, 3.256, 3.456),
    (1, 1024, 1024, 253628, 50, 1.077, 1.115), (1, 1024, 1024, 253628, 200, 4.064, 3.579),
    (1, 1024, 2048, 126567, 200, 2.511, 2.921), (1, 1024, 2048, 126567, 400, 4.611, 5.136),
    (1, 1024, 2048, 253134, 100, 2.149, 2.424), (1, 1024, 2048, 421891, 400, 12.935, 11.647),
    (1, 1024, 2048, 506269, 50, 2.039, 2.227), (1, 1024, 2048, 506269, 400, 15.164, 13.213),
    (1, 2048, 4096, 504792, 200, 9.489, 10.569), (1, 2048, 4096, 504792, 400, 17.366, 19.014),
    (1, 2048, 4096, 1009584, 100, 8.217, 9.802), (1, 2048, 4096, 1009584, 200, 15.997, 17.677),
    (1, 2048, 4096, 1682640, 100, 13.153, 14.107), (1, 2048, 4096, 2019168, 50, 8.050, 9.084),
]


def _records(rules, focused, nx, ny, particles, dt_min, dt_max, learned=0):
    return rules.records_pay(focused, learned, particles, (nx + 4) * (ny + 4), dt_min, dt_max, SMS)


@pytest.mark.parametrize("case", SINGLE, ids=lambda c: "-".join(map(str, c[:5])))
def test_records_of_a_thin_population(rules, case):
    focused, nx, ny, particles, substeps, points_ms, records_ms = case
    dt = (1.0 + 1e-6) / substeps
    picked = records_ms if _records(rules, focused, nx, ny, particles, dt, dt) else points_ms
    assert picked <= 1.02 * points_ms
    if records_ms <= 0.88 * points_ms:
        assert picked == records_ms


def test_records_of_dense_and_small_populations(rules):
    for focused in (0, 1):
        for dt in (0.1, 0.001):
            assert _records(rules, focused, 256, 256, 20000, dt, dt)      # a quarter: always
            assert not _records(rules, focused, 4096, 4096, 60000, dt, dt)  # does not fill the chip
    # adaptive Parker, ms on the point tables / on records
    for nx, ny, particles, points_ms, records_ms in (
            (1024, 2048, 253134, 17.97, 17.06), (1024, 1024, 211356, 15.58, 15.02),
            (1500, 1500, 361922, 51.3, 42.8), (256, 4096, 250510, 71.3, 63.8),
            (256, 4096, 170560, 58.8, 58.3), (1024, 1024, 126814, 11.04, 11.82),
            (1024, 2048, 126567, 11.73, 13.51), (512, 1024, 124655, 2.83, 3.30),
            (512, 1024, 132081, 3.02, 3.44), (700, 800, 133013, 5.31, 6.06),
            (700, 800, 140937, 5.60, 6.26)):
        on = _records(rules, 0, nx, ny, particles, 1e-4, 0.01)
        assert (records_ms if on else points_ms) <= 1.02 * min(points_ms, records_ms)
    # learned closure, ms on the point tables / on records
    for nx, ny, particles, substeps, points_ms, records_ms in (
            (1024, 2048, 421891, 50, 2.129, 2.262), (1024, 2048, 421891, 100, 4.114, 3.967),
            (1024, 2048, 421891, 400, 15.83, 13.84), (1024, 2048, 450000, 50, 2.57, 2.75),
            (1024, 2048, 506269, 50, 2.475, 2.565), (1024, 2048, 506269, 100, 4.807, 4.563),
            (1024, 2048, 506269, 400, 18.53, 16.10), (2048, 4096, 504792, 25, 1.65, 2.80)):
        dt = (1.0 + 1e-6) / substeps
        on = _records(rules, 1, nx, ny, particles, dt, dt, learned=1)
        assert (records_ms if on else points_ms) == min(points_ms, records_ms)


# focused, runs, nx, ny, particles of a run, substeps, and ms of a later
# interval of the batch: on the point tables, on records (fixed steps)
BATCH = [
    (0, 4, 512, 512, 38678, 100, 1.13, 1.15), (0, 4, 512, 512, 38678, 200, 1.98, 1.83),
    (0, 4, 512, 512, 61865, 50, 1.00, 1.08), (0, 4, 512, 512, 77000, 50, 1.15, 1.28),
    (0, 4, 512, 512, 155000, 50, 1.99, 1.87), (0, 4, 512, 512, 155000, 200, 6.60, 4.66),
    (0, 4, 1024, 2048, 168000, 200, 8.10, 8.49), (0, 4, 1024, 2048, 314000, 100, 7.62, 8.24),
    (0, 4, 1024, 2048, 630000, 50, 7.86, 10.02), (0, 4, 1024, 2048, 630000, 100, 14.77, 13.41),
    (0, 4, 1024, 2048, 1250000, 25, 11.22, 14.04), (0, 4, 1024, 2048, 1250000, 50, 15.15, 14.82),
    (0, 16, 512, 512, 62000, 50, 3.26, 3.67), (0, 16, 512, 512, 62000, 100, 5.75, 5.26),
    (0, 16, 512, 512, 156000, 25, 5.37, 6.49), (0, 16, 512, 512, 156000, 50, 7.22, 6.80),
    (0, 16, 1024, 1024, 84000, 100, 8.57, 9.16), (0, 16, 1024, 1024, 252000, 50, 12.63, 16.53),
    (0, 16, 1024, 1024, 314000, 25, 11.08, 16.91), (0, 16, 1024, 1024, 630000, 10, 19.89, 25.15),
    (0, 48, 256, 256, 15600, 100, 4.70, 4.04), (0, 48, 256, 256, 15600, 200, 8.45, 6.57),
    (0, 48, 256, 256, 39400, 25, 4.32, 4.47), (0, 48, 256, 256, 39400, 50, 5.73, 5.14),
    (1, 4, 512, 512, 38678, 100, 1.70, 1.56), (1, 4, 512, 512, 77000, 25, 1.08, 1.10),
    (1, 4, 512, 512, 77000, 50, 1.74, 1.59), (1, 4, 512, 512, 155000, 25, 1.90, 1.82),
    (1, 4, 1024, 2048, 168000, 100, 6.41, 6.62), (1, 4, 1024, 2048, 502000, 50, 9.22, 9.92),
    (1, 4, 1024, 2048, 502000, 100, 17.57, 15.61), (1, 4, 1024, 2048, 630000, 25, 6.99, 9.65),
    (1, 4, 1024, 2048, 630000, 100, 21.88, 18.08), (1, 4, 1024, 2048, 1250000, 50, 22.16, 17.25),
    (1, 16, 512, 512, 62000, 25, 3.00, 3.77), (1, 16, 512, 512, 62000, 100, 9.16, 7.60),
    (1, 16, 512, 512, 156000, 10, 5.42, 6.44), (1, 16, 512, 512, 156000, 50, 11.44, 8.40),
    (1, 16, 1024, 1024, 158000, 50, 11.72, 15.18), (1, 16, 1024, 1024, 252000, 50, 18.29, 19.23),
    (1, 16, 1024, 1024, 314000, 25, 13.74, 18.86), (1, 48, 256, 256, 15600, 100, 7.45, 6.03),
    (1, 48, 256, 256, 39400, 25, 5.58, 5.06), (1, 48, 256, 256, 39400, 50, 9.21, 6.49),
]


@pytest.mark.parametrize("case", BATCH, ids=lambda c: "-".join(map(str, c[:6])))
def test_records_of_a_batch(rules, case):
    focused, runs, nx, ny, particles, substeps, points_ms, records_ms = case
    points = runs * (nx + 4) * (ny + 4)
    total = runs * particles
    on = rules.batch_records_pay(focused, 1, runs, total, points, total * substeps, SMS)
    picked = records_ms if on else points_ms
    # never slower than the quarter rule, and no clear gain left
    assert picked <= 1.02 * (records_ms if 4 * total >= points else points_ms)
    assert picked <= 1.15 * min(records_ms, points_ms)
    # adaptive runs of a dense batch keep their records
    assert rules.batch_records_pay(focused, 0, runs, total, points, total * substeps, SMS) or \
        4 * total < points


# particles of all runs, ms of a fixed-step interval on the point tables with
# 640 and with 384 resident threads per SM, Parker and focused
RESIDENT = [
    (64000, (0.41, 0.46), (0.58, 0.62)),
    (84000, (0.49, 0.54), (0.64, 0.77)), (112000, (0.66, 0.59), (0.90, 0.82)),
    (120000, (0.73, 0.76), (0.99, 1.03)), (160000, (0.87, 0.91), (1.19, 1.26)),
    (188800, (0.96, 1.01), (1.28, 1.48)), (224000, (1.21, 1.16), (1.64, 1.59)),
    (304000, (1.46, 1.46), (1.97, 2.09)), (480000, (1.49, 1.47), (1.88, 1.87)),
    (640000, (2.02, 1.97), (2.60, 2.55)), (980000, (3.60, 3.31), None),
]


@pytest.mark.parametrize("case", RESIDENT, ids=lambda c: str(c[0]))
def test_residency_of_a_batch(rules, case):
    particles, *times = case
    threads = rules.batch_point_threads(particles, 1, 640, SMS)
    assert threads in (640, 384)
    for ms in times:
        if ms is not None:
            assert ms[threads == 384] <= 1.03 * min(ms)
    # adaptive steps, 192 000 particles: 8.97 / 9.40 ms
    assert rules.batch_point_threads(particles, 0, 640, SMS) == 640
    # shapes that hold no more anyway
    assert rules.batch_point_threads(particles, 1, 320, SMS) == 320


# focused (slab QLT), nx, ny, particles, and ms of 100 fixed steps on the point
# tables at 2, 3, 4 and 5 blocks per SM, and at five blocks of an earlier build
# that knew no other residency
POINTS = [
    (0, 512, 1024, 62000, 0.42, 0.47, 0.41, 0.50, 0.51), (0, 512, 1024, 75000, 0.43, 0.53, 0.41, 0.49, 0.51),
    (0, 512, 1024, 95000, 0.62, 0.60, 0.63, 0.49, 0.50), (0, 512, 1024, 110000, 0.62, 0.61, 0.70, 0.74, 0.68),
    (0, 512, 1024, 125000, 0.80, 0.76, 0.76, 0.82, 0.72), (0, 512, 1024, 150000, 0.81, 0.83, 0.79, 0.87, 0.82),
    (0, 512, 1024, 190000, 1.00, 1.05, 1.05, 0.95, 0.96), (0, 512, 1024, 230000, 1.19, 1.18, 1.16, 1.27, 1.18),
    (0, 512, 1024, 300000, 1.55, 1.58, 1.52, 1.57, 1.54), (0, 724, 1448, 62000, 0.47, 0.49, 0.42, 0.51, 0.53),
    (0, 724, 1448, 95000, 0.66, 0.58, 0.67, 0.51, 0.53), (0, 724, 1448, 110000, 0.67, 0.63, 0.69, 0.75, 0.73),
    (0, 724, 1448, 125000, 0.84, 0.78, 0.75, 0.80, 0.77), (0, 724, 1448, 190000, 1.07, 1.07, 1.07, 0.98, 1.00),
    (0, 724, 1448, 230000, 1.27, 1.20, 1.18, 1.29, 1.23), (0, 1024, 2048, 62000, 0.54, 0.57, 0.50, 0.55, 0.56),
    (0, 1024, 2048, 75000, 0.55, 0.58, 0.59, 0.67, 0.69), (0, 1024, 2048, 95000, 0.72, 0.62, 0.80, 0.92, 0.95),
    (0, 1024, 2048, 110000, 0.73, 0.64, 0.81, 1.23, 1.27), (0, 1024, 2048, 125000, 0.90, 0.80, 0.84, 1.19, 1.23),
    (0, 1024, 2048, 150000, 0.92, 0.85, 0.86, 1.09, 1.10), (0, 1024, 2048, 190000, 1.11, 1.09, 1.12, 1.02, 1.06),
    (0, 1024, 2048, 230000, 1.30, 1.22, 1.20, 1.38, 1.31), (0, 1024, 2048, 300000, 1.70, 1.63, 1.58, 1.72, 1.70),
    (1, 512, 1024, 62000, 0.64, 0.71, 0.64, 0.78, 0.79), (1, 512, 1024, 75000, 0.66, 0.74, 0.64, 0.78, 0.79),
    (1, 512, 1024, 95000, 0.94, 0.87, 0.97, 0.78, 0.79), (1, 512, 1024, 110000, 0.95, 0.91, 1.06, 1.11, 1.13),
    (1, 512, 1024, 125000, 1.23, 1.16, 1.20, 1.16, 1.17), (1, 512, 1024, 150000, 1.25, 1.24, 1.22, 1.32, 1.29),
    (1, 512, 1024, 190000, 1.56, 1.60, 1.71, 1.54, 1.53), (1, 512, 1024, 230000, 1.87, 1.77, 1.81, 2.08, 2.16),
    (1, 512, 1024, 300000, 2.45, 2.42, 2.38, 2.73, 2.81), (1, 724, 1448, 62000, 0.77, 0.82, 0.70, 0.79, 0.82),
    (1, 724, 1448, 95000, 1.03, 0.94, 1.10, 0.92, 0.92), (1, 724, 1448, 110000, 1.03, 0.94, 1.15, 1.24, 1.30),
    (1, 724, 1448, 125000, 1.25, 1.20, 1.22, 1.29, 1.28), (1, 724, 1448, 190000, 1.56, 1.63, 1.65, 1.54, 1.57),
    (1, 724, 1448, 230000, 1.88, 1.81, 1.86, 1.98, 2.00), (1, 1024, 2048, 62000, 0.85, 1.10, 0.83, 0.89, 0.91),
    (1, 1024, 2048, 75000, 0.88, 1.08, 1.00, 1.07, 1.02), (1, 1024, 2048, 95000, 1.19, 1.06, 1.47, 1.31, 1.29),
    (1, 1024, 2048, 110000, 1.22, 1.07, 1.47, 1.83, 1.92), (1, 1024, 2048, 125000, 1.47, 1.33, 1.45, 1.81, 1.89),
    (1, 1024, 2048, 150000, 1.50, 1.43, 1.50, 1.82, 1.83), (1, 1024, 2048, 190000, 1.82, 1.72, 1.87, 1.90, 1.91),
    (1, 1024, 2048, 230000, 2.10, 1.88, 1.98, 2.26, 2.27), (1, 1024, 2048, 300000, 2.56, 2.53, 2.53, 2.71, 2.81),
]


@pytest.mark.parametrize("case", POINTS, ids=lambda c: "-".join(map(str, c[:4])))
def test_residency_on_the_point_tables(rules, case):
    focused, nx, ny, particles, *times, earlier = case
    table = 2 * (nx + 4) * (ny + 4) * (96 if focused else 64)
    picked = rules.point_blocks(particles, 1, table, 132644864, SMS)
    assert 2 <= picked <= 5
    ms = times[picked - 2]
    assert ms <= 1.09 * min(times) and ms <= 1.06 * times[1] and ms <= 1.06 * earlier
    assert rules.point_blocks(particles, 0, table, 132644864, SMS) == 3  # adaptive steps
    assert rules.point_blocks(100 * particles, 1, table, 132644864, SMS) == 3


def test_no_launch_leaves_a_preference_on_its_kernel():
    """A kernel's shared-memory share is a property of the process: two threads
    whose launches want different ones would take each other's."""
    with open(os.path.join(CSRC, "kpt_push.cu")) as f:
        assert "cudaFuncAttributePreferredSharedMemoryCarveout" not in f.read()


def test_residency_of_the_fp64_push(rules):
    lanes = 128 * SMS
    # the rule: adaptive one block up to eight populations of its lanes, two
    # beyond; fixed 60 000 particles 10.1 / 7.6 / 8.8 / 7.9 ms, 25 000 5.2 / 3.4 /
    # 4.4 / 5.5 ms with 1 / 2 / 3 / 4 blocks
    assert rules.f64_blocks_per_sm(40000, 0, lanes, 4, 0) == 1
    assert rules.f64_blocks_per_sm(400000, 0, lanes, 4, 0) == 2
    assert rules.f64_blocks_per_sm(60000, 1, lanes, 4, 0) in (2, 4)
    assert rules.f64_blocks_per_sm(25000, 1, lanes, 4, 0) == 2
    # a last round of a few costs a round of their own warps, not of all: focused
    # slab QLT, contracted, 40 steps, two blocks fit, ms with 1 / 2 blocks
    for particles, one, two in ((41000, 5.48, 4.70), (50000, 5.55, 4.84), (58000, 5.61, 5.05),
                                (80000, 8.97, 7.72)):
        picked = rules.f64_blocks_per_sm(particles, 1, lanes, 2, 0)
        assert (one, two)[picked - 1] <= min(one, two)
    # a request is honoured in both directions, up to what fits
    for fixed in (0, 1):
        for particles in (256, 40000, 400000):
            for requested in (1, 2, 3, 4, 9):
                assert rules.f64_blocks_per_sm(particles, fixed, lanes, 4, requested) == \
                    min(requested, 4)
                assert rules.f64_blocks_per_sm(particles, fixed, lanes, 2, requested) == \
                    min(requested, 2)


# the same with one, two, three and five blocks of 128 threads
@pytest.mark.parametrize("particles,parker,focused", [
    (8000, (0.15, 0.18, 0.22, 0.21), (0.20, 0.25, 0.33, 0.27)),
    (16000, (0.17, 0.19, 0.23, 0.26), (0.21, 0.26, 0.33, 0.41)),
    (24000, (0.46, 0.36, 0.44, 0.58), (0.60, 0.48, 0.62, 0.85)),
    (32000, (0.27, 0.22, 0.24, 0.32), (0.34, 0.29, 0.34, 0.46))])
def test_residency_of_a_small_batch(rules, particles, parker, focused):
    picked = {128: 0, 256: 1, 384: 2, 640: 3}[rules.batch_point_threads(particles, 1, 640, SMS)]
    assert parker[picked] == min(parker) and focused[picked] == min(focused)
