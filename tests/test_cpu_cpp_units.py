"""Runs the host-only C++ unit tests of csrc/tests/*.cpp (compile-time loop, prefetch-ring driver, partitioning).

Counterpart of the single-GPU unit binaries csrc/tests/static_for.cu and csrc/tests/pipeline.cu of the reference;
the headers under test are host/device code, so the logic is checked here without a GPU and again inside a kernel
by csrc/tests/device_api_test.cu.
"""
import re
import subprocess
from pathlib import Path


def test_cpu_unit_binary():
    from purlin_b200 import _build
    exes = _build.build_cpu_tests()
    assert exes, "no host-only C++ tests were found"
    for exe in exes:
        res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
        print(res.stdout[-4000:])
        assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-2000:]
        assert "PASSED" in res.stdout and "FAIL " not in res.stdout


def test_arrivals_on_the_other_cta_of_a_pair_name_the_cluster():
    # An arrival from the other CTA hands its tensor memory back to the issuer of the MMAs. Without a scope mbarrier.arrive is of its own
    # CTA only, which the waiter's cluster-scope acquire does not synchronise with; no run shows that, so the instructions are read.
    text = (Path(__file__).resolve().parent.parent / "csrc" / "include" / "purlin" / "tc_sm100.cuh").read_text()
    arrivals = re.findall(r'"(mbarrier\.arrive[\w.:]*)', text)
    remote = [a for a in arrivals if "shared::cluster" in a]
    assert remote and all(re.search(r"\.(release|relaxed)\.cluster\.", a) for a in remote), remote
    waits = re.findall(r'"(mbarrier\.try_wait[\w.:]*)', text)
    assert waits and all(".acquire.cluster." in w for w in waits), waits
