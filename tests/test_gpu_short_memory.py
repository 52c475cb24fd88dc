"""Short device memory, with allocations that are made to fail."""
import os

import pytest

import variant

pytestmark = pytest.mark.gpu


def test_calls_with_failing_allocations(pk_built, tmp_path):
    pytest.importorskip("torch")
    lib = variant.link(str(tmp_path / "libpike_short.so"), [os.path.join(variant.HERE, "short_memory.cpp")],
                       wrap=["cudaMalloc", "cudaMallocFromPoolAsync", "cudaMemPoolTrimTo"])
    variant.run("short_memory_child.py", lib)
