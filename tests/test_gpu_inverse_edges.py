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
