"""The in-place H and E updates (csrc/march.cuh) where their segments, rows and slabs end, against the oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# float64: a few hundred operations' rounding over the steps; float32: the same number of float32 roundings
TOL = {"double": 1e-12, "single": 2e-5}


# x segments of one plane (small grids), of several planes with a remainder, the longest where the CTAs do not fit at
# once (35 planes by 6 in float32; in float64, 22 MB a component, one node per thread); rows shorter than a warp, odd
# rows, rows a CTA holds several of; slabs on one side only, a grid of three planes, periodic axes
@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("shape,pml,periodic", [
    ((7, 9, 5), ((0, 0), (2, 0), (0, 0)), (False, False, False)),
    ((3, 40, 33), ((0, 0), (4, 4), (0, 5)), (True, False, False)),
    ((37, 90, 151), ((6, 5), (5, 0), (7, 6)), (False, False, False)),
    ((41, 131, 97), ((0, 6), (6, 6), (0, 0)), (False, False, True)),
    ((35, 300, 267), ((5, 5), (0, 0), (6, 6)), (False, True, False)),
])
def test_inplace_updates_match_the_oracle(shape, pml, periodic, precision):
    from lightsmith_b200.engine import Engine
    from lightsmith_b200.plan import DFTMonitor, DipoleSource, PMLSpec, flat_index, make_plan
    from oracle.engine import OracleEngine

    rng = np.random.default_rng(5)
    at = [rng.integers(1, n - 1, 400) for n in shape]
    idx = np.unique(flat_index(rng.integers(0, 3, 400), *at, shape))
    src = DipoleSource(idx=idx, coef=rng.normal(size=len(idx)), wave=rng.normal(size=40))
    mon = DFTMonitor(np.array([0.004]), idx[:20], idx[:20], idx[20:40] if len(idx) >= 40 else idx[:20], energy=1)
    kappa = 1.0 if shape[0] != 37 else 3.0
    plan = make_plan(shape=shape, dx=20.0 if shape[0] != 41 else (20.0, 18.0, 22.0), dt=10.0, single=False,
                     inv_eps=1 / rng.uniform(1, 6, shape), groups=[],
                     pml=PMLSpec(cells=pml, alpha_max=0.001, kappa_max=kappa), sources=[src], monitors=[mon],
                     dft_stride=5, periodic=periodic)
    eng, ref = Engine.from_plan(plan, precision=precision, fused=False), OracleEngine(plan)
    assert not eng.fused
    for _ in range(2):
        eng.chunk(1, use_graph=True)
        ref.chunk()
    for a, b in ((eng.E.cpu().numpy(), ref.E), (eng.H.cpu().numpy(), ref.H)):
        assert np.abs(a - b).max() < TOL[precision] * np.abs(b).max()
    eng.close()


# rows shorter than, at and past a tile of the fused pass; a grid past what stays in L2 (188 x 188 x 64 in float64)
@pytest.mark.parametrize("shape,fused", [((24, 21, 28), True), ((24, 21, 32), False), ((19, 40, 68), False),
                                         ((188, 188, 64), True)])
def test_small_grids_step_in_place_with_the_fused_pass_values(shape, fused):
    from lightsmith_b200.engine import Engine
    from lightsmith_b200.plan import DFTMonitor, DipoleSource, PMLSpec, flat_index, make_plan

    rng = np.random.default_rng(6)
    at = [rng.integers(1, n - 1, 300) for n in shape]
    idx = np.unique(flat_index(rng.integers(0, 3, 300), *at, shape))
    src = DipoleSource(idx=idx, coef=rng.normal(size=len(idx)), wave=rng.normal(size=40))
    mon = DFTMonitor(np.array([0.004]), idx[:20], idx[:20], idx[20:40], energy=1)
    plan = make_plan(shape=shape, dx=20.0, dt=10.0, single=False, inv_eps=1 / rng.uniform(1, 6, shape), groups=[],
                     pml=PMLSpec(cells=((4, 5), (6, 0), (5, 5)), alpha_max=0.001), sources=[src], monitors=[mon],
                     dft_stride=5)
    a, b = Engine.from_plan(plan), Engine.from_plan(plan)
    b.set_tuning(4, 8, 0, 4)
    assert a.fused == fused and b.fused
    for e in (a, b):
        for _ in range(3):
            e.chunk(1, use_graph=True)
    for u, v in ((a.E, b.E), (a.H, b.H), (a.monitors[0]["acc_h"], b.monitors[0]["acc_h"])):
        assert (u - v).abs().max() < TOL["double"] * v.abs().max()
    a.close()
    b.close()


# layers that together are as wide as the axis, so that nodes lie in both slabs and take both terms: 3 to 11 shared
# nodes along each axis in turn, one grid with rows shorter than a tile of the fused pass, and a periodic axis
@pytest.mark.parametrize("kappa", [1.0, 3.0])
@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("shape,pml,periodic", [
    ((20, 24, 40), ((10, 10), (4, 4), (5, 5)), (False, False, False)),
    ((22, 17, 37), ((4, 0), (12, 9), (0, 5)), (False, False, False)),
    ((21, 26, 33), ((0, 4), (4, 4), (16, 17)), (False, False, False)),
    ((18, 16, 12), ((0, 0), (8, 8), (6, 6)), (False, False, False)),
    ((16, 12, 36), ((9, 8), (0, 0), (4, 4)), (False, True, False)),
])
def test_overlapping_slabs_add_both_terms(shape, pml, periodic, precision, kappa):
    from lightsmith_b200.engine import Engine
    from lightsmith_b200.plan import DFTMonitor, DipoleSource, PMLSpec, flat_index, make_plan
    from oracle.engine import OracleEngine

    rng = np.random.default_rng(7)
    at = [rng.integers(1, n - 1, 200) for n in shape]
    idx = np.unique(flat_index(rng.integers(0, 3, 200), *at, shape))
    src = DipoleSource(idx=idx, coef=rng.normal(size=len(idx)), wave=rng.normal(size=40))
    mon = DFTMonitor(np.array([0.004]), idx[:20], idx[:20], idx[20:40], energy=1)
    plan = make_plan(shape=shape, dx=20.0, dt=10.0, single=False, inv_eps=1 / rng.uniform(1, 6, shape), groups=[],
                     pml=PMLSpec(cells=pml, alpha_max=0.001, kappa_max=kappa), sources=[src], monitors=[mon],
                     dft_stride=10, periodic=periodic)
    ref = OracleEngine(plan)
    for _ in range(3):
        ref.chunk()
    for fused in (None, False):  # the default choice, and the in-place kernels
        eng = Engine.from_plan(plan, precision=precision, fused=fused)
        for _ in range(3):
            eng.chunk(1, use_graph=True)
        for a, b in ((eng.E.cpu().numpy(), ref.E), (eng.H.cpu().numpy(), ref.H)):
            assert np.abs(a - b).max() < TOL[precision] * np.abs(b).max()
        assert int(eng.n.item()) == 30
        eng.close()


# the choice between the two in-place forms of wide values, on both sides of its lines (8 MB a component, rows that fill
# 0.8 of the lanes): float64 103 x 100 x 95 (7.8 MB), 106 x 100 x 96, the same nodes in rows of 100; complex values in
# Bloch cells; with one 1/eps per component, mirror planes of both signs, cells that are not cubic, slabs at the far
# ends
@pytest.mark.parametrize("shape,dx,pml,bloch,mirror,kappa", [
    ((103, 100, 95), 20.0, ((5, 5), (5, 5), (5, 5)), 0, (0, 0, 0), 1.0),
    ((106, 100, 96), (20.0, 18.0, 22.0), ((5, 5), (5, 5), (5, 5)), 0, (0, 0, 0), 3.0),
    ((106, 96, 100), 20.0, ((5, 0), (0, 5), (5, 5)), 0, (0, 0, 0), 1.0),
    ((30, 31, 200), 20.0, ((0, 0), (0, 0), (8, 8)), 2, (0, 0, 0), 1.0),
    ((75, 75, 190), (20.0, 20.0, 18.0), ((0, 0), (0, 0), (8, 8)), 2, (0, 0, 0), 1.0),
    ((12, 90, 31), 20.0, ((4, 4), (0, 0), (0, 5)), 1, (0, 0, 0), 3.0),
    ((37, 41, 33), 20.0, ((0, 5), (0, 5), (4, 4)), 0, (-1, 1, 0), 1.0),
    ((41, 33, 37), 20.0, ((4, 4), (0, 5), (0, 5)), 0, (0, -1, 1), 1.0),
    ((110, 95, 127), 20.0, ((0, 5), (5, 5), (0, 5)), 0, (1, 0, -1), 3.0),
])
@pytest.mark.parametrize("precision", ["double", "single"])
def test_inplace_forms_match_the_oracle(shape, dx, pml, bloch, mirror, kappa, precision):
    from lightsmith_b200.engine import Engine
    from lightsmith_b200.plan import DFTMonitor, DipoleSource, PMLSpec, flat_index, make_plan
    from oracle.engine import OracleEngine

    rng = np.random.default_rng(8)
    at = [rng.integers(3, n - 1, 300) for n in shape]
    idx = np.unique(flat_index(rng.integers(0, 3, 300), *at, shape))
    periodic = (bloch == 2, bloch > 0, False)
    plan = make_plan(shape=shape, dx=dx, dt=10.0, single=False, groups=[],
                     inv_eps=1 / rng.uniform(1, 6, (3,) + shape),
                     pml=PMLSpec(cells=pml, alpha_max=0.001, kappa_max=kappa), dft_stride=6, periodic=periodic,
                     bloch=tuple(0.004 if p else 0.0 for p in periodic), mirror=mirror,
                     sources=[] if bloch else [DipoleSource(idx=idx, coef=rng.normal(size=len(idx)),
                                                            wave=rng.normal(size=40))],
                     monitors=[DFTMonitor(np.array([0.004]), idx[:20], idx[:20], idx[20:40], energy=1)])
    eng, ref = Engine.from_plan(plan, precision=precision, fused=False), OracleEngine(plan)
    if bloch:  # no point current in complex fields: both start from the same E between the CPML layers
        seed = np.zeros(3 * np.prod(shape), complex)
        seed[idx] = rng.normal(size=len(idx)) + 1j * rng.normal(size=len(idx))
        ref.E[...] = seed.reshape(ref.E.shape)
        eng.E.copy_(eng.E.new_tensor(ref.E))
    for _ in range(2):
        eng.chunk(1, use_graph=True)
        ref.chunk()
    for a, b in ((eng.E.cpu().numpy(), ref.E), (eng.H.cpu().numpy(), ref.H)):
        assert np.abs(a - b).max() < TOL[precision] * np.abs(b).max()
    eng.close()


# a grid that steps in place by its size, asked about and stepped before a kernel is chosen: the choice still holds
@pytest.mark.parametrize("variant", [1, 3, 4])
def test_a_kernel_choice_holds_after_the_default_was_decided(variant):
    from lightsmith_b200.engine import Engine
    from lightsmith_b200.plan import DFTMonitor, DipoleSource, PMLSpec, flat_index, make_plan

    shape = (24, 21, 32)
    rng = np.random.default_rng(9)
    at = [rng.integers(1, n - 1, 300) for n in shape]
    idx = np.unique(flat_index(rng.integers(0, 3, 300), *at, shape))
    src = DipoleSource(idx=idx, coef=rng.normal(size=len(idx)), wave=rng.normal(size=40))
    mon = DFTMonitor(np.array([0.004]), idx[:20], idx[:20], idx[20:40], energy=1)
    plan = make_plan(shape=shape, dx=20.0, dt=10.0, single=False, inv_eps=1 / rng.uniform(1, 6, shape), groups=[],
                     pml=PMLSpec(cells=((4, 5), (6, 0), (5, 5)), alpha_max=0.001), sources=[src], monitors=[mon],
                     dft_stride=5)
    a, b = Engine.from_plan(plan), Engine.from_plan(plan, fused=False)
    assert not a.fused
    a.step(3)
    b.step(3)
    a.set_tuning(variant, 8, 0, 4)
    assert a.fused and not b.fused
    for e in (a, b):
        e.step(2)
        e.sample()
        e.chunk(2, use_graph=True)
    a.check_status()
    for u, v in ((a.E, b.E), (a.H, b.H), (a.monitors[0]["acc_h"], b.monitors[0]["acc_h"])):
        assert (u - v).abs().max() < TOL["double"] * v.abs().max()
    assert int(a.n.item()) == int(b.n.item()) == a.n_host == 15
    a.close()
    b.close()


# the step count, which every step of a call but its last leaves to the next one's H kernel, over every way to advance a
# run, in both in-place forms (float64 overlapping slabs: k_update_nodes); a table source without E corrections writes
# its incident view by itself
@pytest.mark.parametrize("e_points", [True, False])
@pytest.mark.parametrize("pml", [((4, 5), (6, 0), (5, 5)), ((4, 5), (12, 12), (5, 5))])
def test_step_count_over_every_way_to_advance(pml, e_points):
    from lightsmith_b200.engine import Engine
    from lightsmith_b200.plan import DFTMonitor, DipoleSource, PMLSpec, TablePoints, TableSource, flat_index, make_plan
    from oracle.engine import OracleEngine

    shape, m, rows = (24, 21, 27), 3, 60
    rng = np.random.default_rng(10)
    at = [rng.integers(2, n - 2, 60) for n in shape]
    idx = np.unique(flat_index(rng.integers(0, 3, 60), *at, shape))
    table = rng.normal(size=rows)

    def points(k):
        return TablePoints(idx[:k], np.zeros(k, np.int64), rng.integers(0, 20, k), rng.uniform(0, 1, k),
                           rng.normal(size=k))
    view = object()
    src = TableSource(table, np.stack([table, 2 * table, 0 * table]).reshape(-1), m, rows - 6,
                      points(40) if e_points else None, points(30),
                      (rows * np.arange(3), rng.integers(0, 20, 3), rng.uniform(0, 1, 3)), view)
    dip = DipoleSource(idx=idx, coef=rng.normal(size=len(idx)), wave=rng.normal(size=80))
    om = np.array([0.004, 0.011])
    plan = make_plan(shape=shape, dx=20.0, dt=10.0, single=False, inv_eps=1 / rng.uniform(1, 6, shape), groups=[],
                     pml=PMLSpec(cells=pml, alpha_max=0.001), sources=[src, dip], dft_stride=5,
                     monitors=[DFTMonitor(om, idx[:20], idx[:20], idx[20:40], energy=1),
                               DFTMonitor(om, np.arange(3), None, None, energy=0, source=view)])
    eng, ref = Engine.from_plan(plan, fused=False), OracleEngine(plan)
    at = 0

    def check(steps):
        nonlocal at
        for _ in range(steps):
            ref.step()
        at += steps
        assert int(eng.n.item()) == at == eng.n_host
        for a, b in ((eng.E, ref.E), (eng.H, ref.H)):
            assert np.abs(a.cpu().numpy() - b).max() <= TOL["double"] * np.abs(b).max()
    for n in (1, 4, 1, 2):
        eng.step(n)
        check(n)
    for graph in (False, True, True, False):
        eng.chunk(1, use_graph=graph)
        check(5)
        ref.sample()
        eng.step(1)
        check(1)
    eng.chunk_timed(1)
    check(5)
    ref.sample()
    for k, q in enumerate(ref.monitors):
        assert np.abs(eng.results(k)[0] - q["acc_e"]).max() <= TOL["double"] * np.abs(q["acc_e"]).max()
    eng.close()
