"""Sources name no path of the machine they were written on."""
import os

from conftest import ROOT


def test_no_machine_paths():
    bad = []
    for top in ("cemc_gb300", "include", "oracle", "perf", "tests"):
        for folder, dirs, files in os.walk(os.path.join(ROOT, top)):
            dirs[:] = [d for d in dirs if not d.startswith(("_", "."))]
            bad += [os.path.join(folder, f) for f in files
                    if f.endswith((".py", ".sh", ".c", ".cpp", ".cu", ".cuh", ".h"))
                    and "/" + "root/" in open(os.path.join(folder, f)).read()]
    bad += [f for f in ("__graft_entry__.py", "bench.py") if "/" + "root/" in open(os.path.join(ROOT, f)).read()]
    assert not bad
