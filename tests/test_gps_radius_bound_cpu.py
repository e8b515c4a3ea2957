"""The constants behind the error bound of the fast GPS position (gps_limits in csrc/kernels.cu) against the radius
table they describe: its largest step from node to node, and its largest radius."""
import re

import numpy as np

from _parity import lut
from test_pdl_reads_cpu import source


def test_table_steps_and_radii():
    text = source("kernels.cu")
    slope = float(re.search(r"kLutSlope = ([0-9.]+)f", text).group(1))
    radius = float(re.search(r"kGpsEw = kLutSlope \* 1\.3e-4f \+ 4e-6f \+ ([0-9.]+)f \*", text).group(1))
    t = np.asarray(lut(), np.float64).reshape(65, 129)
    step = np.abs(np.diff(t, axis=1)).max()
    assert 0.9 * slope < step <= slope, step
    assert 0.0 <= t.min() and 0.9 * radius < t.max() <= radius, (t.min(), t.max())
