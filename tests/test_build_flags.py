"""Device code stays uncompressed in the library: unpacking it took 25 of the
55 ms of a process's first evaluation.  (The time itself is not tested: on a
shared host it spreads from 30 to 200 ms.)"""
from md_b200 import build


def test_device_code_is_not_compressed():
    assert "--no-compress" in build.FLAGS
