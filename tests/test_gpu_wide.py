"""The wide form of the FP64 kernel (small launches) against the one-pass form, bit for bit, over
tile remainders, tree sizes, mapping kinds, lab boosts, per-event beams and batches."""
import numpy as np
import pytest

from conftest import all_maps_process, wide_beams
from gpu_phs_gb300 import processes as P
from gpu_phs_gb300.philox import uniform_x

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def make(kind):
    if isinstance(kind, int):
        return all_maps_process(40 + kind, kind, 5)
    return {"ww": P.ww, "tt": P.tt, "precision": P.precision,
            "nested": lambda: P.nested_resonances(12)}[kind]()


def same(torch, a, b):
    for u, v in zip((a.p, a.factor, a.volume, a.ok), (b.p, b.factor, b.volume, b.ok)):
        assert torch.equal(u, v)


@pytest.mark.parametrize("kind", ["ww", "tt", "precision", "nested", 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("beams", ["equal", "lab", "event"])
def test_wide_form_equals_one_pass(torch, kind, beams):
    from gpu_phs_gb300.api import PhaseSpace
    proc = make(kind)
    e = 0.5 * (proc.sqrts or 1000.0)
    E1, E2 = (1.2 * e, e / 1.2) if beams == "lab" else (e, e)
    wide, plain = PhaseSpace(proc, E1, E2), PhaseSpace(proc, E1, E2)
    plain.set_variants(-1, 0)
    for n in (1, 31, 33, 1500):
        counts = None
        if proc.n_channels > 1:
            counts = np.bincount(np.arange(n) * 7 % proc.n_channels, minlength=proc.n_channels).astype(np.int64)
        x = torch.from_numpy(uniform_x(500 + n, n, proc.n_x)).cuda()
        x[:, :max(0, proc.n_out - 2)] *= 0.7       # lighter branches: more events pass the test
        if n > 31:
            x[5, :] = 0.0
            x[6, :] = 0.5
            x[7, :] = 0.125
        if beams == "event":
            b = [torch.from_numpy(v).cuda() for v in wide_beams(n, 2 * e, 9)]
            same(torch, wide.generate_beams(x, *b, counts), plain.generate_beams(x, *b, counts))
        else:
            same(torch, wide.generate(x, counts), plain.generate(x, counts))


def test_wide_form_in_a_batch(torch):
    from gpu_phs_gb300.api import Batch, PhaseSpace
    procs, counts = P.batched(11, 12, 3000)
    spaces = [PhaseSpace(p, 0.5 * p.sqrts, 0.5 * p.sqrts) for p in procs]
    wide, plain = Batch(spaces), Batch(spaces)
    plain.set_variants(-1, 0)
    g = torch.Generator(device="cuda").manual_seed(4)
    size = int(sum(p.n_x * int(c) for p, c in zip(procs, counts)))
    x = torch.rand(size, dtype=torch.float64, device="cuda", generator=g)
    for u, v in zip(wide.generate(x, counts), plain.generate(x, counts)):
        assert torch.equal(u, v)


@pytest.mark.parametrize("n_channels", [1, 31, 64, 65, 90])
def test_split_forms_over_many_segments(torch, n_channels):
    """The split forms number their claims in shared memory up to 64 segments and with a scan
    kernel beyond: the one-pass form's bits either way (FP64), its flags (FP32 pairs)."""
    from gpu_phs_gb300.api import PRECISION_F32X2, Batch, PhaseSpace
    procs, counts = P.batched(21, n_channels, 60 * n_channels)
    spaces = [PhaseSpace(p, 0.5 * p.sqrts, 0.5 * p.sqrts) for p in procs]
    g = torch.Generator(device="cuda").manual_seed(n_channels)
    size = int(sum(p.n_x * int(c) for p, c in zip(procs, counts)))
    x = torch.rand(size, dtype=torch.float64, device="cuda", generator=g)
    plain = Batch(spaces)
    plain.set_variants(-1, 0)
    want = plain.generate(x, counts)
    for v in (5, 6, 7, 8):
        split = Batch(spaces)
        split.set_variants(-1, v)
        for _ in range(2):
            for u, w in zip(split.generate(x, counts), want):
                assert torch.equal(u, w)
    for v in (4, 5):
        pairs = Batch(spaces)
        pairs.set_precision(PRECISION_F32X2)
        pairs.set_variants(v, -1)
        assert torch.equal(pairs.generate(x, counts)[3], want[3])
