"""Which kernel an FP64 thin-disk batch renders with (the trace by samples is
the default, a chosen schedule or block size decides otherwise) and what the
autotuner and scarce memory leave behind. The library's host code on a host
stand-in of the CUDA runtime; CPU only."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "grrt_b200", "csrc")
NATIVE = os.path.join(ROOT, "tests", "native")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("batch_choice")
    srcs = [os.path.join(NATIVE, "batch_choice_host.cpp")] + [
        os.path.join(CSRC, f) for f in ("batch.cpp", "context.cpp", "fits.cpp", "host/scene_tables.cpp",
                                        "host/volumetric_tables.cpp")]
    objs = [str(d / (os.path.basename(s) + ".o")) for s in srcs]
    jobs = [subprocess.Popen(["/usr/bin/g++", "-std=c++20", "-O1", "-fno-pie", "-fopenmp", "-I/usr/local/cuda/include",
                              "-c", "-o", o, s]) for s, o in zip(srcs, objs)]
    assert all(j.wait() == 0 for j in jobs)
    exe = str(d / "batch_choice")
    # the launches that these programs do not reach stay unresolved
    subprocess.run(["/usr/bin/g++", "-no-pie", "-fopenmp", "-Wl,--unresolved-symbols=ignore-all", "-o",
                    exe] + objs, check=True)

    def run(*args):
        out = subprocess.run([exe, *args], check=True, capture_output=True, text=True, timeout=120).stdout
        steps = {}
        for line in out.splitlines():
            m = re.match(r"(\w+) rc=(-?\d+)(?: ran=(\w+) schedule=(\S+) block=(\d+) took=(\w+))?$", line)
            if m:
                steps[m[1]] = dict(rc=int(m[2]), ran=m[3], schedule=m[4], block=m[5], took=m[6])
        return steps

    return run


def test_samples_unless_chosen(program):
    assert program("default")["first"]["ran"] == "samples"
    s = program("schedule")["set"]
    assert s["ran"] == "pixels" and s["schedule"] == "256,1,0"  # what a fresh batch reports, set by the caller
    # the mixed form's tolerances do not choose a schedule, another block size does
    assert program("tolerance")["set"]["ran"] == "samples"
    b = program("block")
    assert b["set"]["ran"] == b["back"]["ran"] == "pixels"
    assert program("too_many")["large"]["ran"] == "pixels"


def test_mixed_autotune_leaves_the_fp64_default(program, tmp_path):
    cache = str(tmp_path / "cache.jsonl")
    for what in ("mixed_autotune", "mixed_cached"):  # timed, then from the file
        s = program(what, cache)
        assert s["autotune"]["rc"] == 0 and s["mixed"]["ran"] == "mixed"
        assert s["fp64"]["ran"] == "samples"


def test_fp64_autotune_is_a_choice(program, tmp_path):
    cache = str(tmp_path / "cache.jsonl")
    for what in ("fp64_autotune", "fp64_cached"):
        s = program(what, cache)
        assert s["autotune"]["rc"] == 0
        assert s["fp64"]["ran"] == s["again"]["ran"] == "pixels"


@pytest.mark.parametrize("what", ["failed_autotune", "failed_mixed_autotune"])
def test_failed_autotune_changes_nothing(program, what):
    s = program(what)
    assert s["autotune"]["rc"] == -1
    a = s["after"]
    assert (a["rc"], a["ran"], a["schedule"], a["block"]) == (0, "samples", "256,1,0", "128")


def test_scratch_only_while_there_is_room(program):
    s = program("no_room")
    assert s["full"]["rc"] == 0 and s["full"]["ran"] == "pixels"
    assert s["freed"]["ran"] == s["replay"]["ran"] == "samples"  # asked again, not given up for good
    assert s["freed"]["took"] == "memory" and s["replay"]["took"] == "none"
    # half of what is free is not taken without being asked for
    s = program("little_room")
    assert s["little"]["ran"] == "pixels"
    assert s["asked"]["rc"] == 0 and s["asked"]["ran"] == "samples"
