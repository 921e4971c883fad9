"""The pipelined host call."""
import numpy as np
import pytest

from gpu_phs_gb300 import processes as P
from gpu_phs_gb300.philox import uniform_x

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(1 << 18) - 1, 1 << 18, 300_001, 900_000])
def test_a_call_of_many_events_chooses_the_variant(torch, n, precision):
    """A host call of 2^18 events times the variants, on its first chunk; shorter ones do not; the
    results are the device call's."""
    from gpu_phs_gb300.api import PhaseSpace
    proc = P.ww()
    x = torch.from_numpy(uniform_x(3, n, proc.n_x)).pin_memory()
    ps = PhaseSpace(proc, 250.0, 250.0)
    ps.set_precision(precision)
    h = ps.generate_host(x)
    ff, f64 = ps.tuning()
    chosen, other = (ff, f64) if precision else (f64, ff)
    assert (chosen >= 0) == (n >= 1 << 18) and other == -1
    h2 = ps.generate_host(x)
    d = ps.generate(x.cuda())
    torch.cuda.synchronize()
    for e in (h, h2):
        for a, b in ((e.p, d.p), (e.factor, d.factor), (e.volume, d.volume), (e.ok, d.ok)):
            assert torch.equal(a, b.cpu())


@pytest.mark.parametrize("pinned", ["none", "all", "p", "factor"])
@pytest.mark.parametrize("n", [1000, 40_000, 600_001])
def test_pinned_and_pageable_outputs(torch, n, pinned):
    """Pinned outputs take small chunks first, pageable ones the largest: the same results."""
    from gpu_phs_gb300.api import Events, PhaseSpace
    proc = P.tt()
    x = torch.from_numpy(uniform_x(5, n, proc.n_x)).pin_memory()
    ps = PhaseSpace(proc, 500.0, 500.0)
    d = ps.generate(x.cuda())
    out = []
    for name, shape, dtype in (("p", (n, proc.n_out, 4), torch.float64), ("factor", (n,), torch.float64),
                               ("volume", (n,), torch.float64), ("ok", (n,), torch.uint8)):
        t = torch.full(shape, 7, dtype=dtype)
        out.append(t.pin_memory() if pinned in ("all", name) else t)
    h = ps.generate_host(x, out=Events(*out))
    for a, b in ((h.p, d.p), (h.factor, d.factor), (h.volume, d.volume), (h.ok, d.ok)):
        assert torch.equal(a, b.cpu())
