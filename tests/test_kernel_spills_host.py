"""Registers of the kernels that walk transform tiles in a loop, as the compiler reports them
for sm_100a (no GPU).  Their tile code splits its exchange and twiddle addresses: with whole
addresses the 2^12 tiles spill 100 to 700 bytes a thread and run up to 1.4 times as long."""

from __future__ import annotations

import concurrent.futures as cf
import re
import subprocess

import pytest


def _spills(name: str, tmp) -> dict[str, int]:
    from vfhe_b200.build import ARCH, CSRC, NVCC_FLAGS, nvcc

    r = subprocess.run([nvcc(), *ARCH, *NVCC_FLAGS, "-Xptxas", "-v", "-c", str(CSRC / f"{name}.cu"), "-o",
                        str(tmp / f"{name}.o")], check=True, capture_output=True, text=True)
    found = re.findall(r"entry function '(\S+)'.*?(\d+) bytes spill stores", r.stderr, re.S)
    assert found
    return {k: int(n) for k, n in found}


@pytest.fixture(scope="module")
def spills(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("spills")
    with cf.ThreadPoolExecutor() as ex:
        return dict(kv for d in ex.map(lambda n: _spills(n, tmp), ["worklist", "ntt_flow"]) for kv in d.items())


def test_looping_tile_kernels_do_not_spill_their_addresses(spills):
    def most(pattern: str) -> int:
        hit = [n for k, n in spills.items() if re.search(pattern, k)]
        assert hit, pattern
        return max(hit)

    assert most(r"k_wl_persistentILi0E") <= 272
    assert most(r"k_wl_persistentILi2E") <= 112
    assert most(r"k_flow_fILi12E") <= 32
