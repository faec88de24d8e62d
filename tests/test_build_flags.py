"""The library's device code is stored uncompressed: unpacking it is two thirds
of what the first launch of a process waits for (15 ms, 7 without), and nvcc
compresses by itself once a source passes some size."""
from finess_b200 import build


def test_device_code_is_not_compressed():
    assert "-no-compress" in build.NVCC_FLAGS
