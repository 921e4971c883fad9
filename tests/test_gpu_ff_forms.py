"""The FP32-pair kernels with their form pinned (a small launch that is not pinned takes the wide
FP64 form), and the FP64 one-pass kernel pinned at the sizes of the small fixtures."""
import numpy as np
import pytest

from conftest import (REFCPU_FIXTURES, all_maps_process, assert_within_conditioning, counts_of, golden,
                      load_process, wide_beams)
from gpu_phs_gb300 import processes as P
from gpu_phs_gb300.philox import uniform_x
from oracle import oracle
from test_gpu_ff import check

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


def generate(torch, proc, x, sqrts, counts=None, precision=1, variant=0, beams=None):
    from gpu_phs_gb300.api import PhaseSpace
    ps = PhaseSpace(proc, sqrts / 2, sqrts / 2)
    ps.set_precision(precision)
    ps.set_variants(*((variant, -1) if precision else (-1, variant)))
    xd = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    if beams is None:
        ev = ps.generate(xd, counts)
    else:
        ev = ps.generate_beams(xd, *(torch.from_numpy(b).cuda() for b in beams), counts)
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in (ev.p, ev.factor, ev.volume, ev.ok)]


@pytest.mark.parametrize("precision, variant", [(0, 0)] + [(1, v) for v in FF_FORMS])
@pytest.mark.parametrize("name", REFCPU_FIXTURES)
def test_reference_fixtures_pinned(torch, name, precision, variant):
    z = golden(f"refcpu_{name}")
    proc = load_process(z)
    sq = float(z["sqrts"][0])
    x = uniform_x(int(z["seed"][0]), len(z["ok"]), proc.n_x)
    got = generate(torch, proc, x, sq, counts_of(z["channel"], proc.n_channels), precision, variant)
    check(got, z["p"], z["factor"], z["volume"], z["ok"], sq, 1e-12 if precision == 0 else TOL)


@pytest.mark.parametrize("precision, variant", [(0, 0)] + [(1, v) for v in FF_FORMS])
@pytest.mark.parametrize("n_out", [10, 12])
def test_largest_trees_pinned(torch, n_out, precision, variant):
    proc = P.nested_resonances(n_out)
    counts = np.array([3000, 1, 2999], np.int64)
    x = uniform_x(41, int(counts.sum()), proc.n_x)
    r = oracle.Oracle(proc, 1000.0).generate(x, np.repeat(np.arange(3), counts).astype(np.int32))
    got = generate(torch, proc, x, 1000.0, counts, precision, variant)
    check(got, r.p, r.factor, r.volume, r.ok, 1000.0, 1e-12 if precision == 0 else TOL)


@pytest.mark.parametrize("variant", FF_FORMS)
def test_batch_pinned(torch, variant):
    from gpu_phs_gb300.api import Batch, PhaseSpace
    rng = np.random.default_rng(21)
    procs = [P.random_process(rng, n_out, 1, 1000.0) for n_out in (3, 8, 5, 4, 7, 6)]
    batch = Batch([PhaseSpace(p, 500.0, 500.0) for p in procs])
    batch.set_precision(1)
    batch.set_variants(variant, -1)
    counts = np.array([37, 1000, 64, 333, 95, 2048], np.int64)
    po = batch.offsets(counts)[1]
    xs = [uniform_x(30 + i, int(c), p.n_x) for i, (p, c) in enumerate(zip(procs, counts))]
    xflat = torch.from_numpy(np.concatenate([a.reshape(-1) for a in xs])).cuda()
    p, f, v, ok = (t.cpu().numpy() for t in batch.generate(xflat, counts))
    e = np.concatenate([[0], np.cumsum(counts)])
    for i, proc in enumerate(procs):
        r = oracle.Oracle(proc, 1000.0).generate(xs[i])
        k = slice(e[i], e[i + 1])
        check((p[po[i]:po[i + 1]].reshape(-1, proc.n_out, 4), f[k], v[k], ok[k]), r.p, r.factor, r.volume, r.ok,
              1000.0)


@pytest.mark.parametrize("beams", ["uniform", "mid", "wide"])
@pytest.mark.parametrize("n_out", [4, 7, 8])
def test_every_mapping_pinned(torch, n_out, beams):
    """The pair kernels on every mapping kind, uniform and per-event beams, at the bar of
    test_gpu_parity.test_every_mapping_uniform_beams."""
    proc = all_maps_process(100 + n_out, n_out, 8)
    n = 20_000
    counts = np.full(8, n // 8, np.int64)
    ch = np.repeat(np.arange(8), counts).astype(np.int32)
    x = uniform_x((700 if beams == "uniform" else 200) + n_out, n, proc.n_x)
    E = None
    if beams == "mid":
        rng = np.random.default_rng(n_out)
        E = rng.uniform(300.0, 700.0, n), rng.uniform(300.0, 700.0, n)
    elif beams == "wide":
        E = wide_beams(n, 1000.0, 7)
    E1, E2 = E or (None, None)
    sq = np.full(n, 1000.0) if E is None else 2.0 * np.sqrt(E1 * E2)
    o = oracle.Oracle(proc, 1000.0)
    r = o.generate(x, ch, E1=E1, E2=E2)
    for variant in FF_FORMS if E is None else [0, 1]:
        p, f, v, ok = generate(torch, proc, x, 1000.0, counts, 1, variant, E)
        assert_within_conditioning(p, f, ok, o, x, r, sq, E1, E2, TOL, 1024, channels=ch)
        assert (np.abs(v - r.volume) / r.volume).max() < 1e-15


@pytest.mark.parametrize("n_out, per_visit", [(6, 80), (7, 128)])
def test_line_between_the_wide_form_and_the_pairs(torch, n_out, per_visit):
    """Just below the line an unpinned call has the FP64 kernel's bits, just above it the pairs'."""
    proc = P.nested_resonances(n_out).subset([0])
    line = per_visit * (n_out - 1)
    for tiles, precision in ((line, 0), (line + 1, 1)):
        n = 32 * tiles - 5
        x = uniform_x(8, n, proc.n_x)
        got = generate(torch, proc, x, 1000.0, variant=-1)
        want = generate(torch, proc, x, 1000.0, precision=precision)
        for a, b in zip(got, want):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("variant", FF_FORMS)
def test_exact_events_of_many_small_segments(torch, variant):
    """A warp's exact FP64 walk takes events of any segments together: channels of 3 to 8 particles with
    a STEP map each (no float-float form) and 1 to 7 events give the FP64 kernel's bits."""
    from gpu_phs_gb300.api import Batch, PhaseSpace
    rng = np.random.default_rng(77)
    procs = []
    for i in range(90):
        p = P.random_process(rng, 3 + i % 6, 1, 1000.0)
        p.map_ids = p.map_ids.copy()
        # the largest branch below the root
        code = max((c for c in (p.d1[0, 2 ** p.n_out - 2], p.d2[0, 2 ** p.n_out - 2]) if p.has_children[0, c - 1]))
        p.map_ids[0, code - 1] = P.MAP_STEP_E if i % 2 else P.MAP_STEP_H
        p.map_masses[0, code - 1], p.map_widths[0, code - 1] = 300.0, 30.0
        procs.append(p)
    counts = np.array([1 + i % 7 for i in range(len(procs))], np.int64)
    spaces = [PhaseSpace(p, 500.0, 500.0) for p in procs]
    size = int(sum(p.n_x * int(c) for p, c in zip(procs, counts)))
    x = torch.rand(size, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    plain, pairs = Batch(spaces), Batch(spaces)
    plain.set_variants(-1, 0)
    pairs.set_precision(1)
    pairs.set_variants(variant, -1)
    want, got = plain.generate(x, counts), pairs.generate(x, counts)
    assert 20 < int(want[3].sum()) < len(want[3])
    for a, b in zip(got, want):
        assert torch.equal(a, b)
