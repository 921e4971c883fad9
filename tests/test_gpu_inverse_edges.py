"""Edges of the inverse map."""
import numpy as np
import pytest

from gpu_phs_gb300 import processes as P
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("n_out", [2, 3])
def test_azimuth_of_minus_zero(torch, n_out):
    """p_y = -0 beside p_x > 0: the azimuth is -0, x_phi 0 and not 1, at the root and below it."""
    from gpu_phs_gb300.api import PhaseSpace
    proc = P.process_from_trees([(0, 1) if n_out == 2 else (0, (1, 2))], [{}], [0.0] * (2 + n_out), sqrts=1000.0)
    a = np.linspace(0.1, 3.0, 40)
    p = np.zeros((len(a), n_out, 4))
    p[..., 2] = -0.0
    if n_out == 2:
        p[:, 0] = 500.0 * np.stack([np.ones_like(a), np.sin(a), -0.0 * a, np.cos(a)], -1)
        p[:, 1, 0], p[:, 1, 1], p[:, 1, 3] = p[:, 0, 0], -p[:, 0, 1], -p[:, 0, 3]
    else:
        # particle 0 along x, the two others in the x-z plane
        p[:, 0, :2] = 4000.0 / 9.0
        p[:, 1:, 0], p[:, 1:, 1] = 2500.0 / 9.0, -2000.0 / 9.0
        p[:, 1, 3], p[:, 2, 3] = 1500.0 / 9.0, -1500.0 / 9.0
    n = p.shape[0]
    ok = np.ones(n, np.uint8)
    ps = PhaseSpace(proc, 500.0, 500.0)
    fac, x = ps.inverse(torch.from_numpy(p).cuda(), None, ok=torch.from_numpy(ok).cuda())
    torch.cuda.synchronize()
    x = x.cpu().numpy()[0]
    rx = oracle.Oracle(proc, 1000.0).inverse(p, np.zeros(n, np.int32), ok, n_x=proc.n_x)[1][0]
    phi = n_out - 2 + 2 * np.arange(n_out - 1)
    assert (rx[:, phi] == 0).any()
    # a half turn may come from either side; the origin is 0
    assert np.array_equal(x[:, phi] == 0, rx[:, phi] == 0)
    assert x[:, phi].max() < 1
    assert np.abs(x[:, phi] - rx[:, phi]).max() < 1e-12


@pytest.mark.parametrize("own", [False, True])
@pytest.mark.parametrize("kind, n", [("random", n) for n in (1, 63, 64, 65, 129, 5000, 60_001)] +
                         [("nested", n) for n in (1, 65, 5000, 30_011)])
def test_tiles_give_every_event_the_same_bits(torch, kind, n, own):
    """Each block takes chunks of 64 events from all over the call: the outputs of a call are those of
    three calls over parts of its events, with few ok events and with many."""
    from gpu_phs_gb300.api import PhaseSpace
    if kind == "nested":
        proc = P.nested_resonances(12).subset([0, 1, 0, 0])
    else:
        proc = P.random_process(np.random.default_rng(5), 6, 16)
    nch = proc.n_channels
    counts = np.bincount(np.arange(n) * 7 // 5 % nch, minlength=nch).astype(np.int64)
    chan = np.repeat(np.arange(nch), counts)
    ps = PhaseSpace(proc, 500.0, 500.0)
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.rand((n, proc.n_x), dtype=torch.float64, device="cuda", generator=g)
    ev = ps.generate(x, counts)

    def inverse(a, b):
        c = np.bincount(chan[a:b], minlength=nch).astype(np.int64)
        extra = dict(x=x[a:b].contiguous(), factor=ev.factor[a:b].contiguous()) if own else {}
        return ps.inverse(ev.p[a:b].contiguous(), c, ok=ev.ok[a:b].contiguous(), **extra)

    fac, xo = inverse(0, n)
    assert torch.isfinite(fac[ev.ok == 0]).all() and (own or (fac[ev.ok == 0] == 0).all())
    cut = [0, n // 7, n // 2 + 3 if n > 10 else n // 2, n]
    for a, b in zip(cut, cut[1:]):
        if a < b:
            f2, x2 = inverse(a, b)
            assert torch.equal(fac[a:b].view(torch.int64), f2.view(torch.int64))
            assert torch.equal(xo[:, a:b].contiguous().view(torch.int64), x2.view(torch.int64))
