"""The FP32-pair kernels with their form pinned (a small launch that is not pinned takes the wide
FP64 form)."""
import numpy as np
import pytest

from gpu_phs_gb300 import processes as P
from gpu_phs_gb300.philox import uniform_x

pytestmark = pytest.mark.gpu

TOL = 1e-7             # momenta (to max(E, 1e-3 sqrt(s))) and factors, as in test_gpu_ff.py
FF_FORMS = [0, 3, 5]   # one pass, fused compacting, split (pre-test kernel + walk)


@pytest.fixture(scope="module")
def torch():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def four_tops():
    """pp -> t t t t -> 12 fermions at 13 TeV: eight narrow resonances below two free pairs."""
    def top(k):
        return (k, (k + 1, k + 2))

    tree = ((top(0), top(3)), (top(6), top(9)))
    maps = {}
    for k in (0, 3, 6, 9):
        maps[0b111 << k] = (P.MAP_SCHANNEL, 173.0, 1.5)
        maps[0b110 << k] = (P.MAP_SCHANNEL, 80.419, 2.048)
    return P.process_from_trees([tree], [maps], [0.0, 0.0] + [4.7, 0.0, 0.0] * 4, name="pp_4t_12f",
                                sqrts=13000.0)


def tiny_mapping_mass():
    """Infrared maps of 1e-7 GeV: a0 = 1e-14 GeV^2."""
    proc = P.precision()
    proc.map_masses = np.where(proc.map_ids == P.MAP_INFRARED, 1e-7, proc.map_masses)
    return proc


LARGE = {"tiny_mapping_mass": tiny_mapping_mass,
         "nested_1TeV": lambda: P.nested_resonances(12),
         "nested_3TeV": lambda: P.nested_resonances(12, 3000.0),
         "nested_13TeV": lambda: P.nested_resonances(12, 13000.0),
         "four_tops": four_tops}


@pytest.mark.parametrize("beams", ["uniform", "event"])
@pytest.mark.parametrize("name", LARGE)
def test_factor_of_many_narrow_resonances(torch, name, beams):
    """The product of the mappings' constants, (pi m Gamma / s)^n, lies below the floats' range:
    the factor of every ok event is the FP64 kernel's within the bar, and so are flags and
    momenta."""
    from gpu_phs_gb300.api import PhaseSpace
    proc = LARGE[name]()
    n = 60_000
    e = 0.5 * proc.sqrts
    counts = None if proc.n_channels == 1 else np.array([n // 2, n // 4, n // 4], np.int64)
    x = torch.from_numpy(uniform_x(77, n, proc.n_x)).cuda()
    rng = np.random.default_rng(2)
    b = [torch.from_numpy(rng.uniform(0.9, 1.1, n) * e).cuda() for _ in range(2)]

    def run(ps):
        ev = ps.generate(x, counts) if beams == "uniform" else ps.generate_beams(x, *b, counts)
        torch.cuda.synchronize()
        return ev

    ref = PhaseSpace(proc, e, e)
    ref.set_variants(-1, 0)
    r = run(ref)
    sel = r.ok.bool()
    assert int(sel.sum()) > 500
    floor = torch.clamp(r.p[sel][..., 0].abs(), min=1e-3 * proc.sqrts)
    for variant in FF_FORMS if beams == "uniform" else [0, 1]:
        ps = PhaseSpace(proc, e, e)
        ps.set_precision(1)
        ps.set_variants(variant, -1)
        ev = run(ps)
        assert torch.equal(ev.ok, r.ok)
        assert int((ev.factor[sel] == 0).sum()) == 0
        ferr = ((ev.factor[sel] - r.factor[sel]).abs() / r.factor[sel].abs()).max().item()
        perr = ((ev.p[sel] - r.p[sel]).abs().amax(-1) / floor).max().item()
        print(f"{name} {beams} variant {variant}: ok {int(sel.sum())}, factor {ferr:.2e}, momenta {perr:.2e}")
        assert ferr <= TOL, ferr
        assert perr <= TOL, perr


@pytest.mark.parametrize("n_out, n", [(6, 810_000), (6, 12_000), (8, 77_924), (8, 20_000), (8, 28_700)])
def test_host_call_has_the_device_call_s_form(torch, n_out, n):
    """A host call's chunks (16384 events, then growing, a short last one) take the form of the whole
    call: the device call's bits, where a chunk alone would be small enough for the FP64 wide form
    too.  (28 700 events in three channels: 897 or 898 tiles of 7 visits, just beyond the line.)"""
    from gpu_phs_gb300.api import PhaseSpace
    proc = P.nested_resonances(n_out)
    counts = np.array([n - 2 * (n // 3), n // 3, n // 3], np.int64)
    x = torch.from_numpy(uniform_x(19, n, proc.n_x)).pin_memory()
    ps = PhaseSpace(proc, 500.0, 500.0)
    ps.set_precision(1)
    h = ps.generate_host(x, counts)
    d = ps.generate(x.cuda(), counts)
    torch.cuda.synchronize()
    for a, b in ((h.p, d.p), (h.factor, d.factor), (h.volume, d.volume), (h.ok, d.ok)):
        assert torch.equal(a, b.cpu())
