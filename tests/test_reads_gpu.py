"""Field reads into pinned arrays (written by the kernel itself up to 4 MiB, by the copy engine above) against the
same reads into pageable arrays: the same kernel's values, so equal bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned(shape, skip=0):
    import torch
    t = torch.empty(int(np.prod(shape)) + skip, dtype=torch.float64, pin_memory=True)
    return t[skip:].numpy().reshape(shape, order="F")


@pytest.mark.parametrize("n", [1, 7, 64, 417, 419])  # 24 bytes per node: 4 MiB lies between 418^2 and 419^2
@pytest.mark.parametrize("which", ["both", "rho", "u", "mixed"])
def test_pinned_reads_equal_pageable_reads(lib, n, which):
    import lbmengine as lbm
    rng = np.random.default_rng(n)
    n0 = max(n, 2)
    kw = dict(dims=2, latticeParameter=1.0, relaxationTimeRatio=0.8, xlims=(0.0, n0 - 1.0), ylims=(0.0, float(n)))
    shape = (n0, n + 1)
    m = lbm.modelInit(massDensity=1.0 + 1e-3 * rng.standard_normal(shape),
                      fluidVelocity=1e-3 * rng.standard_normal(shape + (2,)), **kw)
    m.step(3)
    rho, u = np.empty(shape, order="F"), np.empty(shape + (2,), order="F")
    m.read_fields(rho, u)
    prho = _pinned(shape, skip=1) if which != "u" else None
    pu = None if which == "rho" else (np.empty(shape + (2,), order="F") if which == "mixed" else _pinned(shape + (2,)))
    m.read_fields(prho, pu)
    if prho is not None:
        np.testing.assert_array_equal(prho, rho)
    if pu is not None:
        np.testing.assert_array_equal(pu, u)
    m.close()
