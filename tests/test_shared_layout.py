"""Shared-memory structs that are the target of 16-byte asynchronous copies
ask for their alignment themselves: nothing else places them on a 16-byte
boundary when a kernel has other shared variables."""
import subprocess

import pytest

from cauchyfriendly_gb300 import build

SRC = """
#include "mce_chain.cuh"
#include <cstddef>
static_assert(alignof(mce::ChainSmem) % 16 == 0, "the slots are 16-byte aligned");
static_assert(offsetof(mce::ChainSmem, v) % 16 == 0, "the slots come first or padded");
static_assert(mce::kChainPitch % 2 == 0 && mce::kChainRun % 2 == 0, "a run starts on 16 bytes");
"""


def test_chain_slots_are_aligned_for_their_copies(tmp_path):
    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    (tmp_path / "a.cu").write_text(SRC)
    r = subprocess.run([nvcc, "-c", str(tmp_path / "a.cu"), "-o", str(tmp_path / "a.o")] + build._flags(),
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
