"""Which zeta and pressure solver a model runs, and that each of them, and
each way from one to the next, gives the same levels.

Tolerances: a level against the oracle to the parity tolerance, 1e-3 m;
levels of two solvers, which both end on ||r|| <= 1e-8 ||r0|| + 1e-8 in FP64,
to 1e-5 m on regular meshes and 1e-4 m on discs whose elements are fifty
times longer than wide; pressures to 1e-2 of the largest, the tolerance of
the non-hydrostatic parity tests."""
import numpy as np
import pytest

import shygpu
import shyref
from shygpu import cases

pytestmark = pytest.mark.gpu

ZETA_TOL = 1.0e-3


def disc(spokes, rings=4, r0=400.0, dr=100.0, nlv=1, depth=10.0, level=None, **params):
    """Rings of `spokes` nodes around a hub, which is numbered last (its
    neighbours all come before it); one layer with the tide on the outer
    ring, or `nlv` sigma layers, closed, from the start level `level`."""
    ang = 2 * np.pi * np.arange(spokes) / spokes
    rad = r0 + dr * np.arange(rings)
    x = np.r_[(rad[:, None] * np.cos(ang)).ravel(), 0.0]
    y = np.r_[(rad[:, None] * np.sin(ang)).ravel(), 0.0]
    hub = rings * spokes
    node = lambda r, s: r * spokes + s % spokes
    tri = [(hub, node(0, s), node(0, s + 1)) for s in range(spokes)]
    for r in range(rings - 1):
        for s in range(spokes):
            tri += [(node(r, s), node(r + 1, s), node(r + 1, s + 1)), (node(r, s), node(r + 1, s + 1), node(r, s + 1))]
    nen = np.asarray(tri, np.int32) + 1
    nkn, nel = len(x), len(tri)
    hk = depth * (1.0 + 0.1 * np.sin(x / rad[-1] * 2.0))
    c = cases.channel_case(nx=3, ny=3)
    for k in ("czv", "fcorv", "visv", "difv", "tauxnv", "tauynv", "ppv", "rqv", "znv", "utlnv", "vtlnv", "tempv",
              "saltv", "conzv"):
        c.pop(k, None)
    bnd = np.zeros(nkn, np.int32)
    if level is None:
        bnd[node(rings - 1, 0):hub] = 1
    else:
        c["tide"] = np.zeros((0, 1, 4), np.float32)
        c["znv"] = (level * np.cos(np.pi * x / (2 * rad[-1]))).astype(np.float32)
        c["params"] = dict(c["params"], ireib=0)
    if nlv > 1:
        c.update(hlv=-np.arange(1, nlv + 1) / nlv, hldv=np.full(nlv, -1.0 / nlv))
        c["params"] = dict(c["params"], nsigma=nlv)
    c.update(name="disc", nkn=nkn, nel=nel, nlv=nlv, nen3v=nen, xgv=x, ygv=y, hm3v=hk[nen - 1],
             ilhv=np.full(nel, nlv, np.int32), ilhkv=np.full(nkn, nlv, np.int32), bnd_index=bnd,
             params=dict(c["params"], **params))
    return cases._finish(c)


def nh_disc(spokes):
    return disc(spokes, r0=40.0, dr=10.0, nlv=3, depth=15.0, level=0.01, dt=0.2, inohyd=1)


def run(case, n, **opts):
    m = shygpu.Model(case)
    for k, v in opts.items():
        m.set_option(k, v)
    m.set_state_all()
    m.run(n)
    return m


def znv(m, i=0):
    return m.get_state(i, ("znv",))["znv"]


@pytest.mark.parametrize("spokes", [255, 256, 300])
def test_hub_of_more_than_255_neighbours(spokes):
    """The hub's diagonal is the last of its row's entries."""
    c = disc(spokes)
    a, b = run(c, 10), run(c, 10, zeta_tile_rows=512)
    o = shyref.OracleModel(c)
    o.run(10)
    assert np.abs(znv(a) - o.state()["znv"]).max() <= ZETA_TOL
    assert np.abs(znv(a) - znv(b)).max() <= 1.0e-4


@pytest.mark.parametrize("spokes", [250, 300])
def test_pressure_of_a_hub_of_more_than_255_neighbours(spokes):
    c = nh_disc(spokes)
    g = run(c, 5)
    o = shyref.OracleModel(c)
    o.run(5)
    assert np.abs(znv(g) - o.state()["znv"]).max() <= 1.0e-3 * 0.01
    q, (it, _, r0, r) = g.nh(0)
    qo = o.nh()[0]
    assert it > 0 and r <= 1e-8 * r0 + 1e-8
    assert np.abs(q - qo).max() <= 1.0e-2 * np.abs(qo).max()


@pytest.mark.parametrize("variant", [1, 0])
@pytest.mark.parametrize("tile_rows", [0, 512])
def test_plan_made_while_the_default_stream_is_busy(variant, tile_rows):
    """A plan starts from zeroed words and counters whatever another part of
    the program has queued on the default stream meanwhile."""
    import threading
    import torch

    c = cases.channel_case(nx=120, ny=60, lx=150.0 * 119, ly=150.0 * 59)
    want = znv(run(c, 6, zeta_variant=variant, zeta_tile_rows=tile_rows))
    m = shygpu.Model(c)
    m.set_state_all()
    torch.cuda.synchronize()

    def busy():
        for _ in range(60):
            torch.cuda._sleep(8_000_000)                     # 4 ms each, a quarter of a second in all
    t = threading.Thread(target=busy)
    t.start()
    for _ in range(3):
        m.set_option("zeta_variant", variant)
        m.set_option("zeta_tile_rows", tile_rows)
        m.run(2)
    t.join()
    torch.cuda.synchronize()
    assert np.array_equal(znv(m), want)


def test_more_basins_than_a_grid_has_rows():
    """65540 basins in one model (a grid has at most 65535 CTAs in y and z):
    the sums over a basin, of the first, a middle and the last one."""
    cs = [cases.channel_case(nx=3, ny=3, lx=300.0, ly=300.0, seed=s) for s in (1, 2)]
    n = 65540
    m = shygpu.Model([cs[0]] * (n - 1) + [cs[1]])
    for i, c in ((0, cs[0]), (n // 2, cs[0]), (n - 1, cs[1])):
        m.set_state(i)
        a = shygpu.Model(c)
        a.set_state(0)
        assert a.info(0).volume == m.info(i).volume > 0


@pytest.mark.parametrize("nx,ny,opts", [(41, 25, {}), (514, 514, {}), (41, 25, dict(zeta_tile_rows=512)),
                                        (41, 25, dict(zeta_stage=1))])
def test_bounded_waits(nx, ny, opts):
    """A wait for a member (resident: two, and 130, which send their sums
    through member 0) or an arrival (streaming) that does not exist runs out,
    the step reports it, and the same model then runs as if it had not been."""
    c = cases.channel_case(nx=nx, ny=ny, lx=150.0 * (nx - 1), ly=150.0 * (ny - 1))
    ref, m = run(c, 1, **opts), shygpu.Model(c)
    for k, v in opts.items():
        m.set_option(k, v)
    m.set_state(0)
    m.set_option("zeta_barrier_timeout_test", 1)
    with pytest.raises(shygpu.ShyError) as e:
        m.run(1)
    assert e.value.code == 2 and "ran out" in str(e.value)
    m.set_option("zeta_barrier_timeout_test", 0)
    for g in (ref, m):                                       # both clocks have made one step
        g.set_state(0)
        g.run(3)
    assert np.array_equal(znv(m), znv(ref))


def test_levels_across_the_wrap_of_the_launch_number():
    """The resident solver numbers its launches with 16 bits: twelve steps
    across the wrap give the levels that the cluster solver gives."""
    c = cases.channel_case(nx=41, ny=25)
    c["fcorv"] = np.full(c["nel"], 1.0e-4, np.float32)
    m = run(c, 65530)
    ck = m.checkpoint()
    m.run(12)
    a = znv(m)
    m.restore(ck)
    m.set_option("zeta_variant", 0)
    m.run(12)
    assert np.abs(a).max() > 0.01 and np.abs(a - znv(m)).max() <= 1.0e-5


def solvers(m):
    return m.get_option("zeta_variant"), m.get_option("zeta_resident"), m.get_option("nh_resident")


def test_which_solver_runs():
    """The plan each option selects, as get_option tells it."""
    c = cases.channel_case()
    assert solvers(shygpu.Model(c)) == (2, 1, 0)
    rotating = dict(c, fcorv=np.full(c["nel"], 1.0e-4, np.float32))
    for case, opts, want in ((c, dict(zeta_variant=2), (2, 1)), (c, dict(zeta_variant=0), (0, 0)),
                             (c, dict(zeta_tile_rows=512), (2, 0)), (c, dict(zeta_tile_rows=1024), (2, 1)),
                             (c, dict(zeta_stage=1), (2, 0)), (c, dict(symmetric=0), (2, 1)),
                             (rotating, {}, (2, 1)), (rotating, dict(zeta_tile_rows=512), (2, 1)),
                             (rotating, dict(zeta_variant=0), (0, 0))):
        m = shygpu.Model(case)
        for k, v in opts.items():
            m.set_option(k, v)
        assert solvers(m)[:2] == want, opts
    assert solvers(shygpu.Model(cases.seiche_case())) == (2, 1, 1)


def parity(c, g, o):
    a, b = g.get_state(0), o.state()
    assert np.abs(a["znv"] - b["znv"]).max() <= ZETA_TOL
    act = np.arange(c["nlv"])[None, :] < c["ilhkv"][:, None]
    for f in ("tempv", "saltv"):
        assert np.abs(a[f] - b[f])[act].max() <= 1.0e-4 * np.abs(b[f][act]).max(), f


@pytest.mark.parametrize("tile_rows", [128, 512, 2048])
def test_streaming_solver_matches_the_oracle(small3d, tile_rows):
    """The streaming solver with plain loads on the 3D basin (tracers to the
    parity tolerance, 1e-4)."""
    g = run(small3d, 120, zeta_tile_rows=tile_rows)
    assert solvers(g)[:2] == (2, 0) and g.get_option("zeta_stage") == 0
    o = shyref.OracleModel(small3d)
    o.run(120)
    parity(small3d, g, o)
    assert g.info(0).krylov_iters > 0


def test_streaming_solver_in_a_mix():
    """Basins of very different sizes on the streaming solver: the bits that
    each has alone on it, and the resident solver's levels."""
    cs = [cases.basin3d_case(nkn_target=n, nlv=4, seed=s, baroclinic=False, ts=False)
          for n, s in ((50000, 21), (700, 22), (3000, 23))]
    gb = run(cs, 20, zeta_tile_rows=512)
    assert solvers(gb)[:2] == (2, 0)
    for i, c in enumerate(cs):
        assert np.array_equal(znv(run(c, 20, zeta_tile_rows=512)), znv(gb, i)), i
        r = run(c, 20)
        assert solvers(r)[:2] == (2, 1)
        assert np.abs(znv(r) - znv(gb, i)).max() <= 1.0e-5, i


def test_full_ensemble_on_the_streaming_solver():
    """The 64-basin ensemble at its full size: members have the bits that
    they have alone, and the resident solver's levels."""
    ens = cases.ensemble_cases(64)
    g, r = run(ens, 6, zeta_tile_rows=512), run(ens, 6)
    assert solvers(g)[:2] == (2, 0) and solvers(r)[:2] == (2, 1)
    sizes = [c["nkn"] for c in ens]
    for i in (int(np.argmax(sizes)), int(np.argmin(sizes)), 17):
        assert np.array_equal(znv(run(ens[i], 6, zeta_tile_rows=512)), znv(g, i)), i
    for i in range(len(ens)):
        assert np.abs(znv(g, i) - znv(r, i)).max() <= 1.0e-5, i


@pytest.mark.parametrize("coriolis", [0.0, 1.0e-4])
def test_basin_too_wide_for_the_resident_solver(coriolis):
    """313600 rows need more CTAs than the device has resident: the whole
    batch goes to the streaming solver (symmetric) or the clusters."""
    cs = [cases.channel_case(nx=n, ny=n, lx=150.0 * (n - 1), ly=150.0 * (n - 1)) for n in (560, 24)]
    for c in cs:
        c["fcorv"] = np.full(c["nel"], coriolis, np.float32)
    g, ref = run(cs, 3), run(cs, 3, zeta_variant=0)
    assert solvers(g)[:2] == ((2, 0) if coriolis == 0.0 else (0, 0))
    small = run(cs[1], 3)
    assert solvers(small)[:2] == (2, 1)
    assert np.abs(znv(small) - znv(g, 1)).max() <= 1.0e-5
    for i in range(2):
        assert np.abs(znv(g, i) - znv(ref, i)).max() <= 1.0e-5, i


@pytest.mark.parametrize("coriolis", [0.0, 1.0e-4])
def test_share_with_too_many_ghosts(coriolis):
    """A hub of 1400 neighbours: its share would hold more ghosts than a CTA
    has places, so the model runs another solver, and so does a basin beside
    it that would fit."""
    c, other = disc(1400, rings=3, r0=1000.0), cases.channel_case()
    for q in (c, other):
        q["fcorv"] = np.full(q["nel"], coriolis, np.float32)
    g = run([c, other], 5)
    assert solvers(g)[:2] == ((2, 0) if coriolis == 0.0 else (0, 0))
    o = shyref.OracleModel(c)
    o.run(5)
    assert np.abs(znv(g) - o.state()["znv"]).max() <= ZETA_TOL
    assert np.abs(znv(run(other, 5)) - znv(g, 1)).max() <= 1.0e-5


@pytest.mark.parametrize("what", ["hub", "rows"])
def test_pressure_system_that_does_not_fit(what):
    """A share with too many ghosts (a hub of 800 neighbours), or more rows
    (84252) than are resident: the pressure goes to its own device-wide
    solver, for a basin beside it as well."""
    c = nh_disc(800) if what == "hub" else cases.nh_basin_case(nkn_target=7000, lx=600.0, ly=300.0, nlv=12)
    other = cases.seiche_case()
    g, o, alone = run([c, other], 3), shyref.OracleModel(c), run(other, 3)
    o.run(3)
    assert solvers(g)[2] == 0 and solvers(alone)[2] == 1
    z, (q, (it, _, r0, r)), qo = o.state()["znv"], g.nh(0), o.nh()[0]
    assert np.abs(znv(g) - z).max() <= 1.0e-3 * max(np.abs(z).max(), 1.0e-3)
    assert it > 0 and r <= 1e-8 * r0 + 1e-8
    act = np.arange(c["nlv"])[None, :] < c["ilhkv"][:, None]
    assert np.abs(q - qo)[act].max() <= 1.0e-2 * np.abs(qo[act]).max()
    qa, qb = alone.nh(0)[0], g.nh(1)[0]
    assert np.abs(qa - qb).max() <= 1.0e-2 * np.abs(qa).max()
    assert np.abs(znv(alone) - znv(g, 1)).max() <= 1.0e-5


def test_cluster_shape():
    """cluster_size and zeta_threads are kept and told back whatever solver
    runs, hold where clusters solve, and a shape that cannot be is refused."""
    c = cases.channel_case(nx=41, ny=25)
    m = shygpu.Model(c)
    m.set_option("cluster_size", 4)
    shape = lambda m: (m.get_option("cluster_size"), m.get_option("zeta_threads"))
    assert shape(m) == (4, 1024) and solvers(m)[:2] == (2, 1)
    m.set_option("zeta_threads", 256)
    assert shape(m) == (4, 256) and solvers(m)[:2] == (2, 1)
    m.set_state(0)
    m.run(3)
    assert np.array_equal(znv(m), znv(run(c, 3)))
    m.set_option("zeta_variant", 0)
    assert shape(m) == (4, 256) and solvers(m)[:2] == (0, 0)
    a = run(c, 3, zeta_variant=0, zeta_threads=256, cluster_size=4)
    b = run(c, 3, cluster_size=4, zeta_threads=256, zeta_variant=0)
    assert np.array_equal(znv(a), znv(b)) and np.abs(znv(a) - znv(run(c, 3))).max() <= 1.0e-5
    for name, value in (("cluster_size", 3), ("cluster_size", 32), ("zeta_threads", 100), ("zeta_threads", 2048)):
        with pytest.raises(shygpu.ShyError):
            m.set_option(name, value)
    m.set_option("cluster_size", 0)
    assert shape(m) == (1, 1024)
    m.set_option("zeta_variant", 1)
    assert solvers(m)[:2] == (2, 1)


def test_model_bytes_count_the_plan():
    """What shygpu_model_bytes adds for each zeta plan: per row 4 + 4 + 16
    (row, lengths, columns) + 32 (exchange words) bytes resident, 32 + 16 +
    32 + 8 + 32 streaming, and a little more for ghosts, sums and lists."""
    c = cases.channel_case(nx=200, ny=150, lx=150.0 * 199, ly=150.0 * 149)
    n = c["nkn"]
    size = {}
    m = shygpu.Model(c)
    for name, opts in (("resident", {}), ("streaming", dict(zeta_tile_rows=512)), ("clusters", dict(zeta_variant=0)),
                       ("again", dict(zeta_tile_rows=0, zeta_variant=1))):
        for k, v in opts.items():
            m.set_option(k, v)
        size[name] = m.nbytes()
    assert 56 * n <= size["resident"] - size["clusters"] <= 64 * n
    assert 120 * n <= size["streaming"] - size["clusters"] <= 128 * n
    assert size["again"] == size["resident"]


def test_tuned_choices_of_other_plans_are_measured_again(tmp_path):
    """A tune file whose entry names no plans (the options selected other
    solvers then) is not applied; the entry that replaces it is."""
    import os
    import subprocess
    import sys
    import torch

    sm = torch.cuda.get_device_properties(0).multi_processor_count
    f = tmp_path / "tune"
    f.write_text(f"nbasin=1 rows=790 nlv=1 sym=1 cor=0 wd=0 nsc=0 sm={sm}\t"
                 "zeta_stage=0 zeta_tile_rows=512 zeta_variant=2 inner_tol_frac=0.75\n")
    code = ("import shygpu; from shygpu import cases\n"
            "m = shygpu.Model(cases.channel_case()); m.set_state(0)\n"
            "print(m.autotune(steps=2)[1] == -1.0)")
    env = dict(os.environ, SHYGPU_TUNE_FILE=str(f), PYTHONPATH=os.pathsep.join(sys.path))
    out = [subprocess.run([sys.executable, "-c", code], env=env, check=True, capture_output=True,
                          text=True).stdout.split()[-1] for _ in range(2)]
    assert out == ["False", "True"]
    assert len(f.read_text().splitlines()) == 2
