"""Edge cases on the device: the smallest systems, pairs across the periodic
boundary, tiles that are mostly empty, and rejected inputs."""
import numpy as np
import pytest

from conftest import shifted_configuration

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from rumd_b200 import build, capi
    build.build_lib()
    return capi


def pos4_of(xyz, types):
    p = np.zeros((len(xyz), 4), np.float32)
    p[:, :3] = xyz
    p[:, 3] = np.asarray(types, np.int32).view(np.float32)
    return p


def rms_rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


@pytest.mark.parametrize("cutoff", ["SF", "SP", "NS"])
@pytest.mark.parametrize("xyz", [
    [[0.0, 0.0, 0.0], [1.2, 0.0, 0.0]],          # plain pair
    [[-4.5, 0.3, -0.2], [4.7, 0.1, 0.4]],        # pair across the x face (0.8 apart)
    [[4.9, -4.8, 4.7], [-4.6, 4.9, -4.9]],       # across three faces
])
def test_two_particles_against_fp64(capi, oracle, cutoff, xyz):
    params = oracle.lj_params(1, oracle.lj_table())
    box = np.array([10.0, 10.0, 10.0], np.float32)
    pos = pos4_of(xyz, [0, 0])
    e = capi.Engine(device=0, pb=32, tp=1)
    rid = e.add(pos, box, params, 1, cutoff=cutoff)
    e.calc_f()
    f = e.get(rid, "force", 2)
    ref, u, w = oracle.forces_f64(pos[:, :3].astype(np.float64), np.zeros(2, np.int32), box, 1, params,
                                  capi.CUTOFF[cutoff])
    assert np.abs(ref).max() > 0  # the pair interacts
    # the force tolerance (1e-5): a pair 0.7 apart across three faces loses
    # ~1e-6 of its separation to the FP32 subtraction of coordinates near
    # +-L/2, which the r^-13 wall amplifies about 13-fold
    assert rms_rel(f[:, :3].astype(np.float64), ref) < 1e-5
    assert np.allclose(f[0, :3], -f[1, :3], rtol=1e-6, atol=1e-7)  # Newton's third law
    assert abs(e.stats(rid)["pe"] - u.sum()) <= 1e-5 * max(1.0, abs(u.sum()))
    e.close()


@pytest.mark.parametrize("n,tp", [(3, 8), (5, 8), (33, 4), (65, 2)])
def test_tiny_and_ragged_systems(capi, oracle, n, tp):
    """Systems smaller than a tile or a warp, in a small box (fewer than 7
    cells a side: every axis needs the minimum image)."""
    rng = np.random.default_rng(n)
    params = oracle.lj_params(2, oracle.ka_table())
    L = float((n / 0.6) ** (1.0 / 3.0)) + 5.0
    box = np.array([L, L, L], np.float32)
    # random positions at least 0.9 apart
    xyz = []
    while len(xyz) < n:
        c = rng.uniform(-L / 2, L / 2, 3)
        if all(np.linalg.norm((c - q) - L * np.rint((c - q) / L)) > 0.9 for q in xyz):
            xyz.append(c)
    types = rng.integers(0, 2, n)
    pos = pos4_of(np.array(xyz), types)
    e = capi.Engine(device=0, pb=32, tp=tp)
    rid = e.add(pos, box, params, 2, cutoff="SF")
    e.calc_f()
    f = e.get(rid, "force", n)
    ref, u, w = oracle.forces_f64(pos[:, :3].astype(np.float64), types.astype(np.int32), box, 2, params, 2)
    if np.abs(ref).sum() > 0:
        assert rms_rel(f[:, :3].astype(np.float64), ref) < 1e-5
    e.run(50)  # the step loop runs on such systems too
    assert e.stats(rid)["steps"] == 50
    assert np.isfinite(e.get(rid, "pos", n)).all()
    e.close()


def test_rejected_inputs(capi, oracle):
    params = oracle.lj_params(1, oracle.lj_table())
    e = capi.Engine(device=0)
    with pytest.raises(ValueError):
        e.add(pos4_of([[0.0, 0.0, 0.0]], [0]), [10.0, 10.0, 10.0], params, 1)  # one particle
    with pytest.raises(ValueError):
        e.add(pos4_of([[0, 0, 0], [1, 0, 0]], [0, 0]), [10.0, -1.0, 10.0], params, 1)  # bad box
    rid = e.add(pos4_of([[0, 0, 0], [1.1, 0, 0]], [0, 0]), [10.0, 10.0, 10.0], params, 1)
    e.remove(rid)
    with pytest.raises(Exception):
        e.stats(rid)  # removed replica
    e.close()


@pytest.mark.parametrize("req,eff", [((16, 4), (32, 4)), ((48, 1), (64, 1)), ((96, 3), (96, 2)),
                                     ((192, 8), (192, 2)), ((64, 64), (64, 8)), ((128, 16), (128, 4))])
def test_rumd_launch_shapes_are_mapped(capi, oracle, req, eff):
    """RUMD's autotuner shapes (pb 16..192, tp up to 64; Autotune.py:156-158)
    run: pb becomes whole warps and tp one of 1, 2, 4, 8 with pb*tp <= 512,
    and the forces meet the FP64 tolerance."""
    from rumd_b200 import initconf as I
    c = I.ka_config(2000, T=1.0, seed=9)
    params = oracle.lj_params(2, oracle.ka_table())
    e = capi.Engine(device=0, pb=req[0], tp=req[1])
    assert e.launch() == eff
    rid = e.add(c["pos4"], c["box"], params, 2, cutoff="SF")
    e.calc_f()
    f = e.get(rid, "force", 2000)
    e.set_launch(64, 4)
    e.set_launch(*req)
    assert e.launch() == eff
    e.close()
    ref, _, _ = oracle.forces_f64(c["pos4"][:, :3].astype(np.float64), c["types"], c["box"], 2, params, 2)
    assert rms_rel(f[:, :3].astype(np.float64), ref) < 1e-5


@pytest.mark.parametrize("n,box,set_later", [(370, (6.75, 6.75, 6.75), False), (4500, (24.0, 6.75, 23.5), True),
                                             (4500, (6.75, 24.0, 23.5), False)])
def test_coordinates_outside_the_box(capi, n, box, set_later):
    """All-pairs lists (here a side of fewer than five half cut-offs) take any
    image of a coordinate: the forces of the wrapped configuration bit for bit
    (the separations are exact), when a replica is added and when its positions
    are set, and the same images after a run."""
    from rumd_b200 import initconf as I
    params = np.ascontiguousarray(I.lj_params(2, I.KA), np.float32)
    box, types, pos4, out, k = shifted_configuration(n, box, seed=n)
    got = []
    for p in (pos4, out):
        e = capi.Engine(device=0, pb=64, tp=4)
        rid = e.add(pos4 if set_later else p, box, params, 2, cutoff="SF", dt=1e-4, T=0.8)
        if set_later:
            e.calc_f()
            e.set(rid, "pos", p)
        e.calc_f()
        f, st = e.get(rid, "force", n), e.stats(rid)
        assert np.array_equal(e.get(rid, "pos", n), p)
        e.run(2)
        got.append((f, st["pe"], st["virial"], e.get(rid, "pos", n), e.get(rid, "images", n), e.get(rid, "force", n)))
        e.close()
    a, b = got
    assert np.array_equal(a[0], b[0]) and a[1] == b[1] and a[2] == b[2]
    # a coordinate that starts outside is rounded at its larger magnitude once
    # (up to 2.5 boxes: 2^-19), which the stiffest pairs' forces multiply
    assert np.abs(a[3] - b[3])[:, :3].max() < 1e-5
    assert np.array_equal(b[4] - a[4], k)


@pytest.mark.parametrize("persistent", [0, 1])
def test_a_sort_whose_wait_runs_out_is_contained(capi, persistent):
    """The blocks of a sort wait for one that never comes: the call reports it,
    nothing steps with the old list, and the engine goes on from the state
    before; a replica added afterwards is sorted too."""
    from rumd_b200 import initconf as I
    n = 3000
    params = np.ascontiguousarray(I.lj_params(2, I.KA), np.float32)
    conf = [I.ka_config(n, T=1.2, seed=s) for s in (1, 2)]

    def engine():
        e = capi.Engine(device=0, pb=64, tp=2)
        e.set_variant(capi.VARIANT_PERSISTENT, persistent)
        return e, e.add(conf[0]["pos4"], conf[0]["box"], params, 2, T=1.2, vel4=conf[0]["vel4"])

    e, rid = engine()
    e.run(40)
    want = e.get(rid, "pos", n), e.get(rid, "force", n)
    e.close()
    e, rid = engine()
    for call in (e.calc_f, lambda: e.run(5)):
        e.set(rid, "pos", conf[0]["pos4"])  # its list is due
        capi.check(capi.lib().b2md_probe_stall_sort(e._h))
        with pytest.raises(Exception, match="sort"):
            call()
        st = e.stats(rid)
        assert st["steps"] == 0 and st["rebuilds"] == 0 and st["overflow"] == 0
        assert np.array_equal(e.get(rid, "pos", n), conf[0]["pos4"])
    e.run(40)
    got = e.get(rid, "pos", n), e.get(rid, "force", n)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    capi.check(capi.lib().b2md_probe_stall_sort(e._h))
    e.set(rid, "pos", conf[0]["pos4"])
    with pytest.raises(Exception, match="sort"):
        e.calc_f()
    e.remove(rid)
    rid = e.add(conf[1]["pos4"], conf[1]["box"], params, 2, T=1.2, vel4=conf[1]["vel4"])
    e.calc_f()
    f = e.get(rid, "force", n)
    e.close()
    e = capi.Engine(device=0, pb=64, tp=2)
    rid = e.add(conf[1]["pos4"], conf[1]["box"], params, 2, T=1.2, vel4=conf[1]["vel4"])
    e.calc_f()
    assert np.array_equal(e.get(rid, "force", n), f)
    e.close()


def kernel_image(d, L):
    """The minimum image of float32 separations d in a box of length L, with the
    device's float32 operations: the rounding by adding 1.5 * 2^23 (which is none
    far outside the box), the product and sum fused."""
    d, L, m = np.asarray(d, np.float32), np.float32(L), np.float32(12582912.0)
    k = (d * (np.float32(1) / L) + m) - m
    return d.astype(np.float64) - np.float64(L) * k.astype(np.float64)


@pytest.mark.parametrize("far", [False, True])
def test_positions_of_a_blown_up_system_stay_in_the_cell_arrays(capi, far):
    """Coordinates that are infinite or not a number, or far outside the box (a
    system that has blown up), go to some cell of the grid: the evaluation
    returns, and every particle out of their reach, where they were and where
    the device's minimum image puts them, keeps its force."""
    from rumd_b200 import initconf as I
    n, reach = 4000, 2.5 + 0.3 + 0.01
    c = I.ka_config(n, T=0.8, seed=3)
    p = np.ascontiguousarray(I.lj_params(2, I.KA), np.float32)
    e = capi.Engine(device=0, pb=64, tp=2)
    rid = e.add(c["pos4"], c["box"], p, 2, vel4=c["vel4"])
    e.calc_f()
    f0 = e.get(rid, "force", n)
    bad = c["pos4"].copy()
    if far:
        bad[0, 0], bad[1, 1], bad[2, 2], bad[3, :3] = 3e30, -3e30, 5e9, [4e4, -70.0, 1e6]
    else:
        bad[:3, 0] = [np.inf, -np.inf, np.nan]
        bad[3, 1] = bad[3, 2] = np.nan
    e.set(rid, "pos", bad)
    e.calc_f()
    f1 = e.get(rid, "force", n)
    L = c["box"]
    d = c["pos4"][None, :4, :3] - c["pos4"][:, None, :3]
    d -= L * np.rint(d / L)
    keep = ((d * d).sum(-1) > reach ** 2).all(1)
    if far:
        d = np.stack([kernel_image(bad[:, None, k] - bad[None, :4, k], L[k]) for k in range(3)], -1)
        keep &= ((d * d).sum(-1) > reach ** 2).all(1)
    keep[:4] = False
    assert keep.sum() > 3000
    assert np.isclose(f0[keep], f1[keep], rtol=1e-4, atol=1e-3).all()
    e.set(rid, "pos", c["pos4"])
    e.calc_f()
    assert np.array_equal(e.get(rid, "pos", n), c["pos4"])
    assert np.allclose(e.get(rid, "force", n), f0, rtol=1e-4, atol=1e-3)
    e.close()


# (44 bytes a particle, 16 for one field): the largest read in one piece and one
# more; the largest copied out by one thread and one more; an odd size beyond
@pytest.mark.parametrize("n", [35746, 35747, 190650, 190651, 300007, 530003])
def test_read_backs_return_every_particle_in_the_callers_order(capi, n):
    """Positions, velocities and images, known and different for every particle,
    before a sort, after one, and after they have been set anew."""
    from rumd_b200 import initconf as I
    rng = np.random.default_rng(n)
    m = int(np.ceil(np.cbrt(n)))
    box = np.full(3, 1.0625 * m, np.float32)
    sites = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)

    def state():
        pos4 = np.zeros((n, 4), np.float32)
        pos4[:, :3] = (sites[rng.permutation(len(sites))[:n]] + 0.5) * 1.0625 - 0.53125 * m
        vel4 = np.ones((n, 4), np.float32)
        vel4[:, :3] = rng.standard_normal((n, 3))
        return pos4, vel4, rng.integers(-1000, 1000, (n, 3)).astype(np.int32)

    def check(want):
        for got, w in zip(e.read(rid, n), want):
            assert np.array_equal(got, w)
        for name, w in zip(("pos", "vel", "images"), want):
            assert np.array_equal(e.get(rid, name, n), w)

    e = capi.Engine(device=0, max_particles=n, pb=64, tp=2)
    a = state()
    rid = e.add(a[0], box, np.ascontiguousarray(I.lj_params(1, I.LJ), np.float32), 1, vel4=a[1], im3=a[2])
    check(a)
    e.calc_f()
    check(a)
    b = state()
    e.set(rid, "pos", b[0])
    e.set(rid, "vel", b[1])
    e.set(rid, "images", b[2])
    check(b)
    e.calc_f()
    check(b)
    e.close()
