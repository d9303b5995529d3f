"""Field reads into host arrays that are registered with the device in pieces.  The kernel may write an array itself
only where one registration holds all of it; an array with a gap goes to the copy engine, which copies or refuses it,
and the model stays usable."""
from __future__ import annotations

import ctypes as C
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KB = 1024


@pytest.mark.parametrize("pieces,offset", [
    ([(0, 256)], 0),              # one registration, from its first byte
    ([(0, 160)], 0),              # and to its last one
    ([(0, 128), (128, 128)], 8),  # two that touch
    ([(0, 64), (128, 64)], 16),   # two with a gap: both ends of the array registered, its middle not
    ([(0, 64)], 16),              # the end outside
])
def test_reads_into_registered_pieces(lib, pieces, offset):
    import torch

    import lbmengine as lbm
    from lbmengine import _capi as capi
    shape = (160, 128)  # 160 KiB of densities
    m = lbm.modelInit(dims=2, latticeParameter=1.0, relaxationTimeRatio=0.8, xlims=(0.0, 159.0), ylims=(0.0, 127.0),
                      fluidVelocity=1e-3 * np.random.default_rng(0).standard_normal(shape + (2,)))
    m.step(3)
    want = np.empty(shape, order="F")
    m.read_fields(want, None)
    cudart = torch.cuda.cudart()
    block = mmap.mmap(-1, 256 * KB)
    base = C.addressof(C.c_char.from_buffer(block))
    done = []
    try:
        for start, size in pieces:
            assert int(cudart.cudaHostRegister(base + start * KB, size * KB, 2)) == 0  # 2: mapped
            done.append(base + start * KB)
        rho = np.frombuffer(block, dtype=np.float64, count=want.size, offset=offset * KB).reshape(shape, order="F")
        rho[...] = -1.0
        try:
            m.read_fields(rho, None)
            ok = True
        except capi.LbmError:
            ok = False
        whole = len(pieces) == 1 and offset == 0
        assert ok or not whole
        if ok:
            np.testing.assert_array_equal(rho, want)
    finally:
        for p in done:
            cudart.cudaHostUnregister(p)
    again = np.empty(shape, order="F")
    try:
        m.read_fields(again, None)
    except capi.LbmError:  # a refused copy is also the runtime's last error, which the next call may report once
        m.read_fields(again, None)
    np.testing.assert_array_equal(again, want)
    m.close()
