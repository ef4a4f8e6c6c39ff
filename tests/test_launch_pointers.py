"""Kernels launched so that they may start while the kernel before them still runs
(csrc/kernels/launch.cuh): each begins with the wait for it, and takes nothing that a kernel
writes through `const ... __restrict__`, whose loads the compiler may issue as read-only for
the whole life of the kernel, the time before the wait included."""
import glob
import os
import re

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hydrodynamicsgpu_gb300", "csrc",
                       "kernels")
TABLES = ("BatchProblem", "BatchTile")      # copied by the host when a batch is made, never written by a kernel


def dependent_kernels():
    found = {}
    for path in glob.glob(os.path.join(KERNELS, "*.cu")):
        text = open(path).read()
        launched = set(re.findall(r"launchDependent\((\w+)", text))
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\(.*?\)\s+(?=\w+\())?(\w+)\(([^{;]*)\)\s*\{\s*([^;]*;)",
                             text, re.S):
            if m.group(1) in launched:
                found[os.path.basename(path) + ":" + m.group(1)] = (re.sub(r"\s+", " ", m.group(2)), m.group(3))
        missing = launched - {k.split(":")[1] for k in found}
        assert not missing, "%s: no definition found of %s" % (path, sorted(missing))
    return found


def test_wait_comes_first():
    kernels = dependent_kernels()
    assert len(kernels) > 40
    assert [k for k, (_, first) in kernels.items() if first != "dependentLaunch();"] == []


def test_no_read_only_pointers():
    bad = []
    for name, (params, _) in dependent_kernels().items():
        for p in params.split(","):
            if re.search(r"\bconst\b.*__restrict__", p) and not any(t in p for t in TABLES):
                bad.append((name, p.strip()))
    assert bad == []
