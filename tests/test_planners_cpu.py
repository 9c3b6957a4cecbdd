"""Host code of the kernels' planners: small programs print their decisions."""
import math
import os
import shutil
import subprocess

import pytest

import dihydrogen_b200.build as build

import layers

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.skipif(not os.path.exists(build._nvcc()) and shutil.which(build._nvcc()) is None,
                                reason="no nvcc")
FP32, TF32 = 0, 1
MODES = {"fp32": 0, "tf32": 1, "bf16": 3}


def compile_check(folder, name):
    build.build()
    exe = str(folder / name)
    cmd = [build._nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1",
           "-I", os.path.join(ROOT, "include"), "-I", build.CSRC, os.path.join(ROOT, "tests", "cpp", name + ".cu"),
           "-o", exe, "-L", build.PKG, "-ldistconv_b200", "-Xlinker", "-rpath=" + build.PKG]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    exe = compile_check(tmp_path_factory.mktemp("planner"), "conv_planner_check")

    def plan(*geometry):
        r = subprocess.run([exe], input=" ".join(str(v) for v in geometry) + "\n", capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, r.stderr
        return {l.split()[0]: [int(v) for v in l.split()[1:]] for l in r.stdout.splitlines()}

    return plan


@pytest.mark.parametrize("geometry", [
    # n c k d h w f stride: the longest chain of leading products in an accumulator
    (2, 128, 32, 16, 32, 32, 3, 1),   # 216 in one chain
    (2, 256, 16, 16, 32, 32, 3, 1),   # 432
    (8, 128, 32, 0, 56, 56, 5, 1),    # 200
    (8, 256, 256, 0, 14, 14, 3, 1),
    (8, 32, 32, 0, 64, 64, 11, 1),    # 242: the CUDA-core kernel may have it
    (2, 16, 16, 32, 32, 32, 7, 1),
])
def test_chains_of_truncating_updates_are_bounded(planner, geometry):
    plans = planner(*geometry, FP32)
    for name in ("fwd", "bwd_data"):
        ok, chain, nsets, _ = plans[name]
        assert not ok or (0 < chain <= 96 and nsets >= 2), (name, chain, nsets)


@pytest.mark.parametrize("geometry", [
    (1, 16, 32, 64, 64, 64, 3, 2), (8, 64, 128, 0, 56, 56, 3, 2), (1, 32, 32, 24, 40, 67, 3, 1), (2, 32, 32, 0, 96, 131, 5, 2),
    (1, 8, 24, 24, 40, 64, 3, 2),
])
def test_strided_and_wide_layers_are_held_to_the_error_of_fp32_fma(planner, geometry):
    n, c, k, d, h, w, f, s = geometry
    taps = f ** (3 if d else 2)
    most = ((f + s - 1) // s) ** (3 if d else 2)  # of an input cell, backward
    plans = planner(*geometry, FP32)
    assert plans["fwd"][0] == plans["bwd_data"][0] == 1
    # (channels are padded to cells of 8; a chain has at least one update per tap row)
    assert plans["fwd"][1] <= max(0.85 * math.sqrt(c * taps), taps // f), plans
    assert plans["bwd_data"][1] <= max(math.sqrt(k * most), most ** 0.5), plans


@pytest.mark.parametrize("extents", [(1024, 512, 512), (1000, 999, 997)])
def test_large_volumes_are_not_refused(planner, extents):
    """2^28 cells a channel and more (4 -> 16 channels hold 40 to 160 GB in a training step)."""
    plans = planner(1, 4, 16, *extents, 3, 1, FP32)
    assert plans["fwd"][0] == plans["bwd_data"][0] == 1, plans


@pytest.mark.parametrize("extents", [(256, 256, 256), (400, 400, 400), (512, 512, 512), (1024, 512, 512)])
def test_large_volumes_do_not_split_the_filters_of_the_backward_filter(planner, extents):
    """Every role reads, splits and stores all of x again."""
    assert planner(1, 4, 16, *extents, 3, 1, FP32)["bwd_filter"] == [1, 1]


@pytest.mark.parametrize("geometry,simt", [
    # n c k d h w f stride; the CUDA-core kernels take forward, backward data
    ((2, 1, 4, 0, 512, 512, 3, 1), (1, 1)), ((2, 1, 4, 0, 96, 128, 3, 2), (1, 0)), ((2, 4, 8, 0, 512, 512, 3, 1), (1, 0)),
    ((1, 1, 16, 64, 128, 128, 3, 2), (1, 0)), ((1, 8, 4, 64, 128, 128, 3, 2), (0, 1)),
    ((2, 32, 32, 0, 512, 512, 5, 1), (0, 0)), ((4, 16, 16, 0, 64, 64, 3, 1), (0, 0)), ((1, 16, 32, 256, 256, 256, 3, 2), (0, 0)),
    ((1, 1, 4, 64, 128, 128, 3, 1), (0, 0)),
])
def test_layers_of_few_products_take_the_cuda_cores(planner, geometry, simt):
    plans = planner(*geometry, FP32)
    assert (plans["fwd"][3], plans["bwd_data"][3]) == simt, plans


def test_threads_that_look_up_the_encoder_together_all_get_it(tmp_path):
    """A thread that came second used to get none, and with it another kernel."""
    r = subprocess.run([compile_check(tmp_path, "encode_fn_check")], capture_output=True, text=True, timeout=60)
    assert (r.returncode, r.stdout.strip()) == (0, "0"), r.stdout + r.stderr


def test_large_redistributions_are_dealt_out_in_pieces(tmp_path):
    """Above 2e9 cells short runs took a block each, and an extent of 2^32 divided by zero."""
    exe = compile_check(tmp_path, "shuffle_jobs_check")
    jobs = "500 1200 1200 4 1\n64 4294967296 1 1 1\n300 700 100 3 2\n1048576 4096 1 1 1\n"
    r = subprocess.run([exe], input=jobs, capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    lines = [[int(v) for v in l.split()] for l in r.stdout.splitlines()]
    assert len(lines) == 4
    for pieces, most, covered, per_unit in lines:
        assert covered and most < 2000000000 and per_unit >= 1000
    assert lines[2][0] == 1


def test_pieces_of_unaligned_runs_cover_them_once(tmp_path):
    exe = compile_check(tmp_path, "shuffle_pieces_check")
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    good, pairs = map(int, r.stdout.split())
    assert good == pairs > 500


def test_shift_kernel_fetches_zeroed_columns_only(tmp_path):
    """Columns that were fetched with the last block but not zeroed held what an earlier kernel left."""
    r = subprocess.run([compile_check(tmp_path, "shift_columns_check")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    passes, beyond, bad = map(int, r.stdout.split())
    assert passes > 1000 and beyond > 100 and bad == 0, r.stdout


def test_units_of_a_redistribution_are_not_mostly_empty(tmp_path):
    """A run in pieces used to be split by the count of its cells: 2049 of them left half of its units' threads idle."""
    exe = compile_check(tmp_path, "shuffle_units_check")
    r = subprocess.run([exe], input="\n".join(str(n) for n in range(1, 20000, 7)), capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    lines = [[int(v) for v in l.split()] for l in r.stdout.splitlines()]
    assert {way for _, way, _ in lines} == {0, 1, 2}
    # from two units on a run has its own, of which the last may have one access
    assert min(full for _, _, full in lines) >= 66, min((full, way, n) for n, way, full in lines)


def test_tables_that_do_not_fit_leave_a_lower_column(tmp_path):
    """Layouts whose issuers' tables are longer than their argument are passed over; no layer of the other
    tests comes near its 8 KB, so that the limit is lowered here."""
    geometries = [((1, 4, 16, 256, 256, 256, 3, 1), (2048, 1536, 1024, 768, 512)), ((2, 8, 24, 67, 83, 101, 3, 1), (2048, 1024, 768, 512)),
                  ((1, 16, 32, 256, 256, 256, 3, 2), (2048, 1536, 1024, 768)), ((2, 64, 64, 32, 32, 32, 3, 1), (2048, 1536, 1024))]
    exe = compile_check(tmp_path, "shift_tables_check")
    lines = [g + (limit,) for g, limits in geometries for limit in (8192,) + limits]
    r = subprocess.run([exe], input="\n".join(" ".join(map(str, l)) for l in lines), capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    got = [[int(v) for v in l.split()] for l in r.stdout.splitlines()]
    assert len(got) == 2 * len(lines)
    lower = 0
    for i, line in enumerate(lines):
        for tr in range(2):
            ok, size, _, rows, chain, _ = got[2 * i + tr]
            assert ok and size <= line[-1] and 0 < chain <= 96, (line, tr, got[2 * i + tr])
            if line[-1] == 8192:
                full = got[2 * i:2 * i + 2]
            elif full[tr][1] <= line[-1]:
                assert got[2 * i + tr] == full[tr], (line, tr)  # a limit that does not bind changes nothing
            else:
                lower += rows < full[tr][3]
    assert lower >= 8


def test_parts_of_rows_cover_every_output_once(tmp_path):
    """Parts of a row side by side in the lanes, each with its own row blocks or segments; what their outputs read is staged."""
    r = subprocess.run([compile_check(tmp_path, "shift_parts_check")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    passes, parts, bad = map(int, r.stdout.split())
    assert passes > 150 and parts > 30 and bad == 0


def test_windows_that_stay_in_l2_are_unpacked_from_their_start(tmp_path):
    """From the end, a window of 34 to 84 MB cost its tensor's next reader 2 to 7 %: either side of the measured crossing,
    one rank on a device and two."""
    exe = compile_check(tmp_path, "shuffle_from_end_check")
    start, end = (33.6, 67.1, 83.9, 2 * 33.6, 2 * 41.9), (100.7, 134.2, 2 * 58.7, 2 * 134.2)
    r = subprocess.run([exe], input=" ".join(map(str, start + end)), capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == ["0"] * len(start) + ["1"] * len(end)


def test_layers_have_the_layouts_that_the_tests_on_the_gpu_mean(tmp_path):
    exe = compile_check(tmp_path, "conv_layout_check")

    def layout(n, c, k, sp, f, pads, stride, mode):
        flat = len(sp) == 2
        v = [n, c, k, *([0] if flat else []), *sp, *([1] if flat else []), *f, *([0] if flat else []), *pads, stride, MODES[mode]]
        r = subprocess.run([exe], input=" ".join(map(str, v)), capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, r.stderr
        return {l.split()[0]: [int(a) for a in l.split()[1:]] for l in r.stdout.splitlines()}

    for (n, c, k, sp, f, pads), slots in layers.SWEEP:
        for mode in MODES:
            want = slots["fp32" if mode == "fp32" else "bf16"]
            assert layout(n, c, k, sp, f, pads, 1, mode)["sweep"] == [int(want > 0), want], (n, c, k, sp, f, mode)
    for (n, c, k, sp, f, s), passes in layers.ROWS_IN_PARTS:
        for mode in ("fp32", "bf16"):
            got = layout(n, c, k, sp, f, [1] * len(sp), s, mode)
            assert got["sweep"][0] == 0
            in_parts = tuple(p for p in ("fwd", "bwd_data") if got[p][0] and got[p][1] > 1 and got[p][2] > 1)
            assert in_parts == passes[mode], (n, c, k, sp, mode, got)
    n, c, k, sp, f, s = layers.STATISTICS_BY_BULK_STORES
    for mode in ("fp32", "bf16"):
        got = layout(n, c, k, sp, f, [1] * 3, s, mode)
        assert got["sweep"][0] == 0 and got["fwd"][:3] == [1, 1, 1] and got["fwd"][3] > 0, got


def test_no_report_of_a_block_counts_for_another_use_of_it(tmp_path):
    """Filters with one tap along D and one or two along H: an issuer reported blocks that it had not waited for."""
    r = subprocess.run([compile_check(tmp_path, "shift_protocol_check")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    passes, same_step, bad = map(int, r.stdout.split())
    assert passes > 80 and same_step > 30 and bad == 0, r.stdout
