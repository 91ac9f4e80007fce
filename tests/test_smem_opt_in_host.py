"""A kernel's opt-in to more than 48 KB of shared memory is an attribute per device: one
helper keeps it per device, or it is set at every launch (CPU only: the sources)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "temgymcore_gb300", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as fh:
        return fh.read()


@pytest.mark.parametrize("name", ["field_gemm.cu", "trace.cu"])
def test_the_opt_in_is_kept_per_device(name):
    src = _source(name)
    assert "cudaFuncSetAttribute" not in src and "smem_opt_in<" in src


def test_the_helper_keeps_one_bit_a_device():
    body = _source("tg_common.cuh").split("static cudaError_t smem_opt_in", 1)[1].split("\n}", 1)[0]
    assert "cudaGetDevice" in body and re.search(r"1ull << \(dev & 63\)", body)
