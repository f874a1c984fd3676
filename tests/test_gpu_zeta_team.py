"""The resident zeta solver at the edges of its shares and teams, against the
streaming solver and, for rows longer than its fixed block, the oracle.

Both solvers end on ||r|| <= 1e-8 ||r0|| + 1e-8 in FP64, so their levels
agree to the solve tolerance and the rounding of FP32 levels: 1e-5 m, a
hundredth of the parity tolerance, over three steps."""
import numpy as np
import pytest

import shygpu
import shyref
from shygpu import cases

pytestmark = pytest.mark.gpu

TOL = 1.0e-5


def basin(nx, ny, seed=3):
    return cases.channel_case(nx=nx, ny=ny, lx=150.0 * (nx - 1), ly=150.0 * (ny - 1), seed=seed)


def levels(case, n=3, **opts):
    m = shygpu.Model(case)
    for k, v in opts.items():
        m.set_option(k, v)
    m.set_state_all()
    m.run(n)
    return [m.get_state(i)["znv"] for i in range(len(m.cases))], m


# one thread's rows, one CTA's, the first row of the next; the last team of
# small shares and the first of large ones (12288 rows); a one-hop team of
# 20 members, one polled by two warps (36 members) and
# one wider than 128 members
@pytest.mark.parametrize("nx,ny", [(3, 3), (19, 27), (57, 9), (32, 32), (41, 25), (205, 10), (33, 64),
                                   (128, 96), (129, 96), (360, 200), (514, 514)])
def test_resident_solver_matches_streaming(nx, ny):
    case = basin(nx, ny)
    (za,), a = levels(case)
    (zb,), b = levels(case, zeta_tile_rows=512)
    assert a.get_option("zeta_variant") == 2 and b.get_option("zeta_variant") == 2
    assert a.info(0).krylov_iters > 0
    assert np.abs(za - zb).max() <= TOL


@pytest.mark.parametrize("nx,ny", [(3, 3), (57, 9), (41, 25), (205, 40), (257, 160)])
def test_resident_bicgstab_matches_clusters(nx, ny):
    """Coriolis: the non-symmetric system, against the cluster solver."""
    case = basin(nx, ny)
    case["fcorv"] = np.full(case["nel"], 1.0e-4, np.float32)
    (za,), a = levels(case)
    (zb,), b = levels(case, zeta_variant=0)
    assert a.get_option("zeta_variant") == 2 and b.get_option("zeta_variant") == 0
    assert np.abs(za - zb).max() <= TOL


@pytest.mark.parametrize("nx,ny", [(33, 9), (161, 33)])
def test_resident_wetting_and_drying_matches_clusters(nx, ny):
    """The repeat loop inside one CTA and inside a team: the same dry
    elements and vertex levels as the cluster solver's."""
    case = cases.flat_case(nx=nx, ny=ny, lx=200.0 * (nx - 1), ly=200.0 * (ny - 1))
    out = []
    for variant in (1, 0):
        m = shygpu.Model(case)
        m.set_option("zeta_variant", variant)
        m.set_state(0)
        m.run(30)
        out.append((m.wetdry(0), m.get_state(0)["zenv"]))
    assert (out[0][0][0] != 0).any()
    for a, b in zip(out[0][0], out[1][0]):
        assert np.array_equal(a, b)
    assert np.abs(out[0][1] - out[1][1]).max() <= TOL


def test_basin_keeps_its_bits_in_a_batch():
    cs = [basin(57, 9, 1), basin(205, 40, 2), basin(3, 3, 3), basin(300, 150, 4)]
    batch, _ = levels(cs)
    for c, z in zip(cs, batch):
        (alone,), _ = levels(c)
        assert np.array_equal(alone, z)


@pytest.mark.parametrize("spokes", [8, 9, 14])
def test_rows_longer_than_the_block(spokes):
    """A disc of rings around a hub: the hub's row has `spokes` off-diagonal
    entries, the block eight."""
    rings, r0 = 40, 200.0
    ang = 2 * np.pi * np.arange(spokes) / spokes
    x, y = [0.0], [0.0]
    for r in range(1, rings + 1):
        x += list(r0 * r * np.cos(ang))
        y += list(r0 * r * np.sin(ang))
    node = lambda r, s: 1 + (r - 1) * spokes + s % spokes
    tri = [(0, node(1, s), node(1, s + 1)) for s in range(spokes)]
    for r in range(1, rings):
        for s in range(spokes):
            tri += [(node(r, s), node(r + 1, s), node(r + 1, s + 1)), (node(r, s), node(r + 1, s + 1), node(r, s + 1))]
    nen = np.asarray(tri, np.int32) + 1
    nkn, nel = len(x), len(tri)
    c = cases.channel_case(nx=3, ny=3)
    bnd = np.zeros(nkn, np.int32)
    bnd[node(rings, 0):] = 1
    for k in ("czv", "fcorv", "visv", "difv", "tauxnv", "tauynv", "ppv", "rqv", "znv", "utlnv", "vtlnv", "tempv",
              "saltv", "conzv"):
        c.pop(k, None)
    hk = 10.0 + np.sin(np.asarray(x) / 900.0)
    c.update(name="disc", nkn=nkn, nel=nel, nen3v=nen, xgv=np.asarray(x), ygv=np.asarray(y), hm3v=hk[nen - 1],
             ilhv=np.ones(nel, np.int32), ilhkv=np.ones(nkn, np.int32), bnd_index=bnd)
    c = cases._finish(c)
    (z,), _ = levels(c, n=20)
    (zs,), _ = levels(c, n=20, zeta_tile_rows=512)
    o = shyref.OracleModel(c)
    o.run(20)
    assert np.abs(z - zs).max() <= TOL
    assert np.abs(z - o.state()["znv"]).max() <= TOL
