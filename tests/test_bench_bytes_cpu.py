"""The byte floor of bench.py's roofline counts what a particle launch has to read, not how wide the present
record is: per list entry its 8 bytes and the 96 bytes of a splat's record that settle nearly every particle."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402


def test_particle_and_geometry_bytes():
    f = bench.algorithmic_bytes_per_launch
    assert f("particles", 0, 1, 1, 1, 1) == 8 + 96
    assert f("particles", 1, 0, 1, 1, 1) == 8
    assert f("geometry", 0, 0, 1, 1, 1) == 64 + 180 + 96 + 8 + 16
