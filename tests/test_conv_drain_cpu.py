"""A block of the TMA-fed kernels that gave a wait up waits for its own copies before it exits, whichever role gave
up and when: the producer may have issued its last copy and left before another role's wait runs out. In
the source, the drain comes after the block's last barrier, where every role has ended."""
import os

import pytest

from test_pdl_reads_cpu import function, source


@pytest.mark.parametrize("kernel", ["k_conv3", "k_conv_dw"])
def test_drain_after_the_last_barrier(kernel):
    _, body = function(source("conv3x3.cu"), kernel)
    at = body.rindex("__syncthreads()")
    assert body.count("drain_copies(") == 1 and body.index("drain_copies(") > at, kernel
    assert "if (s_abort" in body[at:]
    assert body.rindex("tma_load4(") < at and body.rindex("tcgen05.dealloc") > at
