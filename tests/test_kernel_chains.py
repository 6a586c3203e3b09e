"""Kernels that start before the one ahead of them has finished (grid_chain)
read what the chain writes by plain loads only: of their parameters, just the
tables made with a correlator are __restrict__ or read by __ldg.  (What goes
wrong otherwise depends on where a compiler places a load, so it is held on the
source.)"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "fftcorr_b200", "csrc")
TABLES = {"tabx", "taby", "tabz", "tw", "ktab", "rtab", "items", "folds"}
KERNEL = re.compile(r"__global__[^;{}]*?\b(k_\w+)\s*\(([^{}]*)\)\s*\{([^\n]*\n[^\n]*)")


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def _read(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


@pytest.mark.parametrize("name", _sources())
def test_chained_kernels_read_by_plain_loads(name):
    for kernel, params, body in KERNEL.findall(_read(name)):
        if "grid_chain()" not in body:
            continue
        restricted = set(re.findall(r"__restrict__\s+(\w+)", params))
        assert restricted <= TABLES, (kernel, restricted - TABLES)


def test_the_passes_and_histograms_are_found():
    text = "".join(_read(n) for n in ("fc_fused.cu", "fc_fused_gen.cuh", "fc_hist.cu"))
    chained = [k for k, _, body in KERNEL.findall(text) if "grid_chain()" in body]
    assert len(chained) == len(re.findall(r"^  grid_chain\(\);", text, re.M)) >= 18


@pytest.mark.parametrize("name", ["fc_fused.cu", "fc_fused_gen.cuh", "fc_hist.cu"])
def test_read_only_loads_are_of_tables(name):
    assert set(re.findall(r"__ldg\(&(\w+)", _read(name))) <= TABLES
