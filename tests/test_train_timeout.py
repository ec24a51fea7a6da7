"""Training when a tensor-core kernel reports a timeout or a launch fails: the
run ends soon, gives no losses, leaves no work behind on any stream, and the
next run is sound. The library's host code on a host stand-in of the CUDA
runtime; CPU only."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "grrt_b200", "csrc")
NATIVE = os.path.join(ROOT, "tests", "native")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("train_timeout")
    srcs = [os.path.join(NATIVE, "train_timeout_host.cpp")] + [
        os.path.join(CSRC, f) for f in ("surrogate.cpp", "context.cpp", "fits.cpp", "host/scene_tables.cpp",
                                        "host/volumetric_tables.cpp")]
    objs = [str(d / (os.path.basename(s) + ".o")) for s in srcs]
    jobs = [subprocess.Popen(["/usr/bin/g++", "-std=c++20", "-O1", "-fno-pie", "-fopenmp", "-I/usr/local/cuda/include",
                              "-c", "-o", o, s]) for s, o in zip(srcs, objs)]
    assert all(j.wait() == 0 for j in jobs)
    exe = str(d / "train_timeout")
    # the launches that these programs do not reach stay unresolved
    subprocess.run(["/usr/bin/g++", "-no-pie", "-fopenmp", "-Wl,--unresolved-symbols=ignore-all", "-o", exe] + objs,
                   check=True)

    def run(*args):
        out = subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True, timeout=120).stdout
        steps = {}
        for m in re.finditer(r"^(bad|after) rc=(-?\d+) steps=(\d+) filled=(\d+) last=(\S+) drained=(\d) error=(.*)$",
                             out, re.M):
            steps[m[1]] = dict(rc=int(m[2]), steps=int(m[3]), filled=int(m[4]), last=float(m[5]), drained=m[6] == "1",
                               error=m[7])
        return steps

    return run


# steps of the run, and of those that may run at most after a timeout in the
# third: the first rate's (half the run, in pieces of 256) and one piece more
@pytest.mark.parametrize("steps,most", [(24, 15), (80, 50), (8000, 512)])
def test_a_timeout_ends_the_run(program, steps, most):
    s = program("timeout", steps)
    assert s["bad"]["rc"] == -1 and "timeout" in s["bad"]["error"]
    assert s["bad"]["steps"] <= most and s["bad"]["filled"] == 0 and s["bad"]["drained"]
    a = s["after"]
    assert a["rc"] == 0 and a["steps"] == a["filled"] == steps and a["error"] == "none"
    assert a["last"] == s["bad"]["steps"] + steps  # the losses of this run


@pytest.mark.parametrize("what", ["launch", "eager"])
def test_a_failed_launch_leaves_nothing_behind(program, what):
    s = program(what, 40)
    assert s["bad"]["rc"] == -1 and s["bad"]["filled"] == 0 and s["bad"]["drained"]
    assert s["after"]["rc"] == 0 and s["after"]["filled"] == 40


@pytest.mark.parametrize("steps", [1, 2, 7, 8, 600])
def test_every_step_runs_once(program, steps):
    a = program("eager", steps)["after"]
    assert a["rc"] == 0 and a["steps"] == a["filled"] == steps and a["drained"]
