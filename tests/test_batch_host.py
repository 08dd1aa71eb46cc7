"""A batch's buffers and captured graphs, on the CPU.

The host code of libfk (csrc/fk_engine.cu, as nvcc compiles it) linked with a
runtime that runs on plain memory (native/fake_cuda.cpp): copies are made,
captures recorded and replayed, and every use of a buffer that has been freed
is counted.
"""

import pathlib
import re
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
NATIVE = ROOT / "tests" / "native"
CUDA = pathlib.Path("/usr/local/cuda")


@pytest.fixture(scope="module")
def batch_check(tmp_path_factory):
    import build as fkbuild
    tmp = tmp_path_factory.mktemp("batch")
    obj = fkbuild.OBJ / "fk_engine.o"      # the library's own, when current
    if not obj.exists() or any(s.stat().st_mtime > obj.stat().st_mtime
                               for s in fkbuild.sources()):
        obj = tmp / "fk_engine.o"
        subprocess.run([fkbuild.NVCC, *fkbuild.FLAGS, "-c", "-o", str(obj),
                        str(fkbuild.CSRC / "fk_engine.cu")], check=True,
                       capture_output=True)
    exe = tmp / "batch_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(CUDA / "include"),
                    "-o", str(exe), str(NATIVE / "batch_check.cpp"),
                    str(NATIVE / "fake_cuda.cpp"), str(obj)], check=True)

    def check(name):
        out = subprocess.run([str(exe), name], capture_output=True, text=True,
                             timeout=300)
        assert out.returncode == 0 and out.stdout == f"{name} ok\n", \
            out.stdout + out.stderr
    return check


def test_graphs_hold_no_freed_buffer(batch_check):
    """A graph is replayed only while every buffer it was captured with is
    still there: runs of other sizes, eager and not, between two of it."""
    batch_check("growth")


def test_a_graph_is_captured_once(batch_check):
    """The result's length changes no address that the graph holds, and
    results around the length that is read back at once are whole."""
    batch_check("once")


def test_a_failed_call_is_reported_once(batch_check):
    batch_check("error_once")


def test_a_failed_allocation_fails_one_run(batch_check):
    """Whichever buffer cannot grow, that run alone fails: the next has every
    buffer it uses."""
    batch_check("failed_growth")


def test_dickson_lists_up_to_what_their_offset_holds(batch_check):
    """n = 3 below 8.6e7: 4.4 million primes' residues, 1.75e7 entries when
    each list is filled up to a multiple of four."""
    batch_check("long_lists")


def test_the_bytes_copied_back_are_counted(batch_check):
    batch_check("read_back")


def test_stage_times_cover_their_launches(batch_check):
    batch_check("stage_times")


def test_a_replayed_graph_has_its_own_statistics(batch_check):
    batch_check("replay_stats")


def test_the_tuner_tries_no_grid_twice(batch_check):
    """classify_ctas_per_sm: no value searched launches the default's grid or
    another's, and values that launch the same grid share a graph."""
    import fk_tune
    types = (ROOT / "first-knowns_b200" / "csrc" / "fk_types.h").read_text()
    most = int(re.search(r"kClassCtas = (\d+)", types).group(1))
    grids = [min(v, most)
             for v in fk_tune.SPACE["classify_ctas_per_sm"] + [8]]
    assert len(set(grids)) == len(grids)
    batch_check("class_grids")


def test_which_sieve_a_lone_item_takes(batch_check):
    batch_check("lone_items")


def test_item_buffers_do_not_grow_up_to_a_thousand_items(batch_check):
    batch_check("steady_items")
