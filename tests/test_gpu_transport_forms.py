"""Forms of the transport kernels that a rule on the parameters selects,
against the general form on the same basin."""
import numpy as np
import pytest

import shygpu
from shygpu import cases

pytestmark = pytest.mark.gpu


def run(case, n, **over):
    m = shygpu.Model(case, **over)
    m.set_state_all()
    m.run(n)
    return m.get_state(0), m.info(0).istot


@pytest.mark.parametrize("nlv", [2, 5, 9, 17, 30, 32])
def test_stability_index_without_vanishing_terms(nlv):
    """Implicit vertical terms and no horizontal diffusion: the index from
    the horizontal flows alone equals the general one (reached with a
    diffusivity too small to change an FP32 bit of the flows).  The tracers
    agree to FP32 rounding of the transport's differences: 1e-6 of the
    largest value."""
    case = cases.lagoon_case(nkn_target=700, nlv=nlv, ntracer=2, dt=120.0)
    case["rqv"][case["nkn"] // 2] = 50.0          # an inflow enters the index too
    lean, na = run(case, 6)
    general, nb = run(case, 6, chpar=1.0e-30)
    assert na == nb and na >= 1
    assert np.abs(lean["conzv"] - general["conzv"]).max() <= 1.0e-6 * np.abs(general["conzv"]).max()


@pytest.mark.parametrize("nx,ny", [(3, 3), (64, 64), (65, 64), (300, 260)])
def test_chunked_reduction(nx, ny):
    """Volume and budget of basins of less than a chunk, one, one and a node
    more, and many, alone and in a batch (the same bits)."""
    c = cases.channel_case(nx=nx, ny=ny, lx=150.0 * (nx - 1), ly=150.0 * (ny - 1))
    other = cases.channel_case(nx=80, ny=60)
    a, b = shygpu.Model(c), shygpu.Model([other, c])
    for m in (a, b):
        m.set_state_all()
        m.run(3)
    ia, ib = a.info(0), b.info(1)
    assert ia.volume == ib.volume and ia.volume_budget == ib.volume_budget and ia.dtime == ib.dtime == 180.0
    s = a.get_state(0)
    area = np.zeros(c["nkn"])
    ev = shygpu.set_ev(c)
    np.add.at(area, c["nen3v"].ravel() - 1, np.repeat(4.0 * ev[:, 9].astype(np.float64), 3))
    want = (s["hdknv"][:, 0].astype(np.float64) * area).sum()
    assert abs(ia.volume - want) <= 1e-6 * want   # FP32 areas and products


@pytest.mark.parametrize("make,nlv,over", [
    ("lagoon", 17, {}), ("lagoon", 31, {}), ("lagoon", 32, dict(ilin=0)), ("basin3d", 17, {}), ("basin3d", 20, {}),
    ("basin3d", 25, dict(ahpar=1.0)), ("basin3d", 32, dict(ilin=0, ihwadv=1))])
def test_long_columns_by_thread_match_warp_segments(make, nlv, over):
    """Columns of 17 to 32 layers, whole and cut by the bottom, by Thomas
    sweeps in shared memory against the warp segment's cyclic reduction:
    both FP32, so transports agree to 1e-5 of the largest after one step
    (two orders under the parity tolerance)."""
    case = (cases.lagoon_case(nkn_target=500, nlv=nlv) if make == "lagoon"
            else cases.basin3d_case(nkn_target=700, nlv=nlv))
    case["visv"][:, 1:nlv] = 1.0e-2
    rng = np.random.default_rng(nlv)
    act = np.arange(nlv)[None, :] < case["ilhv"][:, None]
    case["utlnv"] = (0.2 * rng.standard_normal(act.shape) * act).astype(np.float32)
    case["vtlnv"] = (0.2 * rng.standard_normal(act.shape) * act).astype(np.float32)
    out = []
    for threads in (1, 0):
        m = shygpu.Model(case, **over)
        m.set_option("column_threads", threads)
        m.set_state_all()
        m.run(1)
        out.append(m.get_state(0))
    for f in ("utlnv", "vtlnv"):
        scale = max(np.abs(out[1]["utlnv"]).max(), np.abs(out[1]["vtlnv"]).max())
        assert np.abs(out[0][f] - out[1][f]).max() <= 1.0e-5 * scale, f
    assert np.abs(out[0]["znv"] - out[1]["znv"]).max() <= 1.0e-5


@pytest.mark.parametrize("nlv", [4, 9, 20, 32])
@pytest.mark.parametrize("n", [1, 2, 3, 4])
def test_scalars_as_one_group_match_a_partial_group(n, nlv):
    """n tracers that fill the node kernel's right-hand sides against the
    same tracers among five (an instance of ten, partly empty): the same
    sums in the same order, 1e-6 of the largest value."""
    case = cases.lagoon_case(nkn_target=500, nlv=nlv, ntracer=5, dt=60.0)
    few = dict(case)
    few["conzv"] = np.ascontiguousarray(case["conzv"][:n])
    few["params"] = dict(case["params"], nconz=n)
    a, na = run(few, 4)
    b, nb = run(case, 4)
    assert na == nb
    assert np.abs(a["conzv"] - b["conzv"][:n]).max() <= 1.0e-6 * np.abs(b["conzv"]).max()


def test_scalars_with_their_own_substep_counts():
    """Two diffusivities, so two sub-step counts: each scalar as in a model
    that transports it alone."""
    case = cases.basin3d_case(nkn_target=600, nlv=12, baroclinic=False)
    both, nb = run(case, 4, thpar=0.0, shpar=5.0e4)
    only_s, ns = run(case, 4, itemp=0, shpar=5.0e4)
    only_t, nt = run(case, 4, isalt=0, thpar=0.0)
    assert ns > nt and nb == ns
    assert np.abs(both["saltv"] - only_s["saltv"]).max() <= 1.0e-6 * np.abs(both["saltv"]).max()
    assert np.abs(both["tempv"] - only_t["tempv"]).max() <= 1.0e-6 * np.abs(both["tempv"]).max()


@pytest.mark.parametrize("make,nlv,over", [
    ("lagoon", 32, {}), ("basin3d", 17, {}), ("basin3d", 20, dict(nzadapt=3, ibarcl=0)), ("basin3d", 32, dict(nzadapt=32, ibarcl=0)),
    ("hybrid", 26, {})])
def test_long_columns_final_state_by_thread(make, nlv, over):
    """Thickness, levels and transports after the zeta solve of columns of
    17 to 32 layers (sigma, z, hybrid, z-adaptive) by a thread per column
    against a warp segment per column, from the same start: the level of the
    two runs differs by FP32 rounding, so thickness and transports agree to
    1e-5 of the largest."""
    case = (cases.lagoon_case(nkn_target=500, nlv=nlv) if make == "lagoon" else
            cases.hybrid_lagoon_case(nkn_target=500, nsigma=nlv - 8) if make == "hybrid" else
            cases.basin3d_case(nkn_target=700, nlv=nlv))
    assert 16 < case["nlv"] <= 32
    out = []
    for threads in (1, 0):
        m = shygpu.Model(case, **over)
        m.set_option("column_threads", threads)
        m.set_state_all()
        m.run(2)
        out.append(m.get_state(0))
    for f in ("utlnv", "vtlnv", "hdknv", "hdenv"):
        scale = np.abs(out[1][f]).max()
        if f in ("utlnv", "vtlnv"):
            scale = max(np.abs(out[1]["utlnv"]).max(), np.abs(out[1]["vtlnv"]).max())
        assert np.abs(out[0][f] - out[1][f]).max() <= 1.0e-5 * scale, f
    assert np.abs(out[0]["znv"] - out[1]["znv"]).max() <= 1.0e-5


def test_checkpoint_keeps_the_places_of_version_1():
    """A checkpoint holds the places of the arrays that version 1 had and the
    model no longer keeps (zeros), whatever they hold on loading."""
    case = cases.basin3d_case(nkn_target=700, nlv=20)
    n, nel, nlv, nsc = case["nkn"], case["nel"], case["nlv"], 2
    m = shygpu.Model(case)
    m.set_state_all()
    m.run(3)
    ck = np.array(m.checkpoint(), copy=True).view(np.uint8)
    count = int(ck[12:16].view(np.int32)[0])
    sizes = ck[40:40 + 8 * count].view(np.int64)
    start = 40 + 8 * count + np.r_[0, np.cumsum(sizes)]
    assert start[-1] == ck.size
    for gone in ([16 * n, 16 * n, 8 * (n + 2)], [12 * nel * nlv * nsc, 12 * nel * nlv]):
        at = [i for i in range(count - len(gone) + 1) if list(sizes[i:i + len(gone)]) == gone]
        assert len(at) == 1
        a, b = start[at[0]], start[at[0] + len(gone)]
        assert not ck[a:b].any()
        ck[a:b] = 0x7f
    m.run(3)
    want = m.get_state(0)
    m.restore(ck)
    m.run(3)
    got = m.get_state(0)
    for f in ("znv", "utlnv", "tempv"):
        assert np.array_equal(got[f], want[f]), f
