"""The status of every launch in the chain of dependent launches reaches the caller: launch_chain
clears the CUDA error it reports, so a caller that drops its result reports success after a launch
that did not run (a Runge-Kutta stage would then be formed from the last call's Fp)."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "vfs-geophysics-3.1_b200", "csrc")


def _sources():
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            src = re.sub(r"/\*.*?\*/", "", f.read(), flags=re.S)
        yield name, re.sub(r"//[^\n]*", "", src)


def test_no_launch_status_is_dropped():
    calls = 0
    for name, src in _sources():
        for m in re.finditer(r"\blaunch_chain\s*\(", src):
            before = src[:m.start()].rstrip().rstrip("\\").rstrip()
            if before.endswith("int"):  # the definition
                continue
            calls += 1
            assert re.search(r"(\breturn|=|\?|[^:]:)$", before), "%s: %s" % (name, src[m.start():m.start() + 90])
    assert calls > 20


def test_single_kernel_launchers_return_their_status():
    seen = set()
    for name, src in _sources():
        for kind, fn in re.findall(r"\b(void|int)\s+(launch_(?!chain|projection)\w+)\s*\(\s*Ctx\s*\*", src):
            assert kind == "int", "%s: %s drops its launch status" % (name, fn)
            seen.add(fn)
        for m in re.finditer(r"\b(launch_(?:face_flux|fp|rhs)|face_fluxes)\s*\(\s*c\s*\)", src):
            before = src[:m.start()].rstrip()
            assert re.search(r"(\breturn|=|\?|[^:]:)$", before), "%s: %s" % (name, src[m.start():m.start() + 60])
    assert {"launch_face_flux", "launch_fp", "launch_rhs"} <= seen
