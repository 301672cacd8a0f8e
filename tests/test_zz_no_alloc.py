"""The allocation-free force entry point (b2md_forces_noalloc).

It exists for callers that cannot allocate device memory while they call the
library: a host program that owns all device buffers and only lends a plugin
pointers, or a real-time loop that must not call cudaMalloc/cudaFree (they can
synchronise the device and take unbounded time).  The caller passes its own
device buffers; the library's only scratch is a fixed array in its device
image.  Here the test owns the buffers (allocated through torch, as such a
host program would), and the results must equal those of the engine's
b2md_calc_f on the same configuration, within the force tolerance used
throughout the tests (rms relative error <= 1e-5), on two calls in a row.
The comparison runs for every cut-off method (each packs the pair rows
differently), once on a cubic and once on a non-cubic box.

This file is collected last so that a run stopping at its first failure has
already run every other test.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MAX_N = 65536
# (cut-off method, particles, box stretch per axis): the stretch keeps the
# volume, so the density stays 1.2
CASES = [("SF", 4000, (1.0, 1.0, 1.0)), ("SP", 1000, (1.25, 0.9, 1.0 / (1.25 * 0.9))),
         ("NS", 1000, (0.9, 1.2, 1.0 / (0.9 * 1.2)))]


def _melted_ka(capi, initconf, n, cutoff, stretch):
    c = initconf.ka_config(n, T=2.0, seed=4)
    params = initconf.lj_params(2, initconf.KA)
    box = (c["box"] * np.asarray(stretch, np.float32)).astype(np.float32)
    pos4 = c["pos4"].copy()
    pos4[:, :3] *= np.asarray(stretch, np.float32)
    e = capi.Engine(device=0, pb=64, tp=4)
    rid = e.add(pos4, box, params, 2, cutoff=cutoff, vel4=c["vel4"])
    e.run(300)
    e.calc_f()
    out = dict(pos4=e.get(rid, "pos", n), force=e.get(rid, "force", n), stats=e.stats(rid),
               box=np.ascontiguousarray(box, np.float32), params=params)
    e.close()
    return out


def _call(lib, pos_ptr, n, box, params, cutoff, force_ptr, sums_ptr, stream):
    return lib.b2md_forces_noalloc(pos_ptr, n, box.ctypes.data_as(ctypes.c_void_p), 2,
                                   params.ctypes.data_as(ctypes.c_void_p), cutoff, force_ptr, sums_ptr, stream)


@pytest.mark.parametrize("cutoff,n,stretch", CASES)
def test_noalloc_forces_equal_engine_forces_on_two_calls(cutoff, n, stretch):
    import torch
    from rumd_b200 import capi, initconf
    ref = _melted_ka(capi, initconf, n, cutoff, stretch)
    lib = capi.lib()
    dev = torch.device("cuda:0")
    pos = torch.from_numpy(ref["pos4"]).to(dev)
    stream = ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
    params = np.ascontiguousarray(ref["params"], np.float32)
    f_ref = ref["force"].astype(np.float64)
    for call in range(2):
        force = torch.full((n, 4), float("nan"), dtype=torch.float32, device=dev)
        sums = torch.zeros(2, dtype=torch.float64, device=dev)
        rc = _call(lib, ctypes.c_void_p(pos.data_ptr()), n, ref["box"], params, capi.CUTOFF[cutoff],
                   ctypes.c_void_p(force.data_ptr()), ctypes.c_void_p(sums.data_ptr()), stream)
        assert rc == capi.B2MD_OK, lib.b2md_last_error()
        torch.cuda.synchronize(dev)
        f = force.cpu().numpy().astype(np.float64)
        s = sums.cpu().numpy()
        rms = np.sqrt(((f[:, :3] - f_ref[:, :3]) ** 2).sum() / (f_ref[:, :3] ** 2).sum())
        assert rms <= 1e-5, (cutoff, call, rms)
        assert np.abs(f[:, 3] - f_ref[:, 3]).max() < 1e-4, (cutoff, call)
        pe, vir = ref["stats"]["pe"], ref["stats"]["virial"]
        assert abs(s[0] - pe) <= 1e-5 * abs(pe), (cutoff, call, s[0], pe)
        assert abs(s[1] - vir) <= 1e-5 * abs(vir) + 1e-3, (cutoff, call, s[1], vir)


def _brute_force(pos4, box, params, cutoff):
    """FP64 minimum-image pair sum of the valid types: [n, 4] and (U, W)."""
    r = pos4[:, :3].astype(np.float64)
    t = pos4[:, 3].view(np.int32)
    ok = (t >= 0) & (t < 2)
    p = params.reshape(2, 2, 12).astype(np.float64)
    L = box.astype(np.float64)
    out, w = np.zeros((len(r), 4)), 0.0
    for i in np.flatnonzero(ok):
        d = r[i] - r
        d -= L * np.rint(d / L)
        d2 = (d * d).sum(1)
        q = p[t[i]][np.where(ok, t, 0)]
        j = np.flatnonzero((d2 < q[:, 0] ** 2) & ok & (np.arange(len(r)) != i))
        d, d2, q = d[j], d2[j], q[j]
        i2, rc, sc, uc = 1.0 / d2, q[:, 0], q[:, 10], q[:, 11]
        i6 = i2 ** 3
        s = i6 * i2 * (12.0 * q[:, 1] * i6 + 6.0 * q[:, 2])
        u = i6 * (q[:, 1] * i6 + q[:, 2])
        if cutoff == "SF":
            s, u = s - sc / np.sqrt(d2), u + sc * (np.sqrt(d2) - rc) - uc
        out[i, :3], out[i, 3] = (d * s[:, None]).sum(0), 0.5 * u.sum()
        w += (d2 * s).sum()
    return out, ok, w / 6.0


# (particles, box, spread): the last sizes of the one-, two- and four-particle
# all-pairs forms, the first of the cell form, a box too thin for cells, a
# cluster and a droplet that crowd their cells (all pairs again), one that
# does not, and positions several box lengths outside
EDGES = [(2, (9, 9, 9), "all"), (33, (9, 9, 9), "all"), (2400, (13, 13, 13), "all"), (2401, (13, 13, 13), "all"),
         (2999, (14, 14, 13), "all"), (3000, (14, 14, 13), "all"), (3001, (40, 11, 6.2), "all"),
         (3100, (15, 13, 17.5), "outside"), (3500, (400, 390, 410), "cluster"),
         (3500, (400, 390, 410), "droplet"), (3501, (120, 110, 125), "droplet"), (4801, (36, 36, 6), "all")]


@pytest.mark.parametrize("n,lengths,spread", EDGES)
def test_noalloc_forms_against_fp64_sums(n, lengths, spread):
    """The form that a size and box select, with particles of unknown type
    among them (NaN forces, no pairs), against FP64 sums; two calls agree bit
    for bit.  Bound: the force tolerance of the tests above."""
    import torch
    from rumd_b200 import capi, initconf
    rng = np.random.default_rng(n)
    box = np.array(lengths, np.float32)
    side = {"cluster": 14.0, "droplet": 46.0}.get(spread)
    ext = box.astype(np.float64) if side is None else np.full(3, side)
    if n == 2:
        ext = np.full(3, 2.0)  # in range of each other
    m = np.maximum(1, np.ceil(ext * (n / ext.prod()) ** (1 / 3) * 1.08)).astype(int)
    while m.prod() < n:
        m[np.argmin(m / ext)] += 1
    g = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3)
    sites = g[rng.permutation(len(g))[:n]]
    pos = (sites + 0.5 + rng.uniform(-0.1, 0.1, (n, 3))) * (ext / m) - ext / 2
    if spread == "outside":
        pos += rng.integers(-2, 3, (n, 3)) * box
    types = (rng.random(n) < 0.2).astype(np.int32)
    if n == 2:
        types[:] = 0
    if n > 100:
        types[rng.integers(0, n, 3)] = [2, -1, 77]
    pos4 = np.zeros((n, 4), np.float32)
    pos4[:, :3] = pos
    pos4[:, 3] = types.view(np.float32)
    params = np.ascontiguousarray(initconf.lj_params(2, initconf.KA), np.float32)
    ref, ok, W = _brute_force(pos4, box, params, "SF")
    lib = capi.lib()
    dev = torch.device("cuda:0")
    p = torch.from_numpy(pos4).to(dev)
    got = []
    for _ in range(2):
        force = torch.zeros((n, 4), dtype=torch.float32, device=dev)
        sums = torch.zeros(2, dtype=torch.float64, device=dev)
        rc = _call(lib, ctypes.c_void_p(p.data_ptr()), n, box, params, capi.CUTOFF["SF"],
                   ctypes.c_void_p(force.data_ptr()), ctypes.c_void_p(sums.data_ptr()),
                   ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
        assert rc == capi.B2MD_OK, lib.b2md_last_error()
        torch.cuda.synchronize(dev)
        got.append((force.cpu().numpy(), sums.cpu().numpy()))
    assert np.array_equal(got[0][0], got[1][0], equal_nan=True) and np.array_equal(got[0][1], got[1][1])
    f, s = got[0]
    assert np.isnan(f[~ok]).all() and np.isfinite(f[ok]).all()
    err = np.linalg.norm(f[ok, :3] - ref[ok, :3]) / np.linalg.norm(ref[ok, :3])
    assert err <= 1e-5, err
    assert abs(s[0] - ref[ok, 3].sum()) <= 1e-5 * np.abs(ref[ok, 3]).sum()
    assert abs(s[1] - W) <= 1e-5 * np.abs(ref[ok, :3]).sum()


@pytest.mark.parametrize("pairs", [300, 1250, 2100])
def test_noalloc_shifted_force_term_is_the_engines(pairs):
    """Particles in isolated pairs, in all three forms, of a table without
    repulsion and attraction: forces and energies are the shifted-force terms
    c/r and c r alone, which must be the engine's bit for bit (1/r refined)."""
    import torch
    from rumd_b200 import capi, initconf
    rng = np.random.default_rng(pairs)
    n, m = 2 * pairs, int(np.ceil(pairs ** (1 / 3)))
    box = np.full(3, 6.0 * m, np.float32)
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:pairs]
    u = rng.standard_normal((pairs, 3))
    u *= rng.uniform(0.85, 2.6, (pairs, 1)) / np.linalg.norm(u, axis=1, keepdims=True)
    x = (g + 0.5) * 6.0 - 3.0 * m + rng.uniform(-0.4, 0.4, (pairs, 3))
    pos4 = np.zeros((n, 4), np.float32)
    pos4[:, :3] = np.concatenate([x - u / 2, x + u / 2])[rng.permutation(n)]
    pos4[:, 3] = (rng.random(n) < 0.3).astype(np.int32).view(np.float32)
    params = np.ascontiguousarray(initconf.lj_params(2, initconf.KA), np.float32)
    params.reshape(-1, 12)[:, 1:3] = 0.0  # A12, A6
    params.reshape(-1, 12)[:, 10:] = rng.uniform(0.5, 1.5, (4, 2))  # s(rc) rc, u(rc)
    e = capi.Engine(device=0, pb=64, tp=4)
    rid = e.add(pos4, box, params, 2, cutoff="SF")
    e.calc_f()
    want = e.get(rid, "force", n)
    e.close()
    dev = torch.device("cuda:0")
    p = torch.from_numpy(pos4).to(dev)
    force = torch.zeros((n, 4), dtype=torch.float32, device=dev)
    sums = torch.zeros(2, dtype=torch.float64, device=dev)
    rc = _call(capi.lib(), ctypes.c_void_p(p.data_ptr()), n, box, params, capi.CUTOFF["SF"],
               ctypes.c_void_p(force.data_ptr()), ctypes.c_void_p(sums.data_ptr()),
               ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
    assert rc == capi.B2MD_OK
    torch.cuda.synchronize(dev)
    assert np.count_nonzero(want[:, 3]) > n // 2
    assert np.array_equal(force.cpu().numpy(), want)


def test_noalloc_overlapping_calls_stay_in_their_outputs():
    """Calls that share the scratch because nothing orders them have undefined
    results, but write only their own outputs, and leave the next call right."""
    import torch
    from rumd_b200 import capi, initconf
    lib, dev, pad = capi.lib(), torch.device("cuda:0"), 4096
    params = np.ascontiguousarray(initconf.lj_params(2, initconf.KA), np.float32)
    calls = []
    for n, T in ((65521, 1.0), (3000, 1.0), (30011, 1.0)):
        c = initconf.ka_config(n, T=T, seed=n)
        calls.append(dict(n=n, box=np.ascontiguousarray(c["box"], np.float32), pos=torch.from_numpy(c["pos4"]).to(dev),
                          out=torch.full((n + 2 * pad, 4), 7.0, device=dev),
                          sums=torch.zeros(2, dtype=torch.float64, device=dev), stream=torch.cuda.Stream(dev)))

    def launch(c):
        rc = _call(lib, ctypes.c_void_p(c["pos"].data_ptr()), c["n"], c["box"], params, capi.CUTOFF["SP"],
                   ctypes.c_void_p(c["out"][pad:].data_ptr()), ctypes.c_void_p(c["sums"].data_ptr()),
                   ctypes.c_void_p(c["stream"].cuda_stream))
        assert rc == capi.B2MD_OK

    torch.cuda.synchronize(dev)
    want = []
    for c in calls:
        launch(c)
        torch.cuda.synchronize(dev)
        want.append(c["out"].clone())
    for _ in range(30):
        for c in calls:
            launch(c)
    torch.cuda.synchronize(dev)
    for c in calls:
        assert (c["out"][:pad] == 7.0).all() and (c["out"][pad + c["n"]:] == 7.0).all()
    for c, w in zip(calls, want):
        launch(c)
        torch.cuda.synchronize(dev)
        assert torch.equal(c["out"], w)


def test_noalloc_rejects_sizes_beyond_its_maximum():
    from rumd_b200 import capi
    lib = capi.lib()
    box = np.array([10.0, 10.0, 10.0], np.float32)
    params = np.zeros(12, np.float32)
    dummy = ctypes.c_void_p(16)  # never dereferenced: the size check comes first
    rc = lib.b2md_forces_noalloc(dummy, MAX_N + 1, box.ctypes.data_as(ctypes.c_void_p), 1,
                                 params.ctypes.data_as(ctypes.c_void_p), 0, dummy, dummy, None)
    assert rc == capi.B2MD_ERR_ARG
    assert str(MAX_N).encode() in lib.b2md_last_error()


def test_noalloc_rejects_cutoffs_beyond_half_the_box():
    from rumd_b200 import capi, initconf
    lib = capi.lib()
    params = np.ascontiguousarray(initconf.lj_params(1, initconf.LJ), np.float32)  # rc = 2.5
    dummy = ctypes.c_void_p(16)  # never dereferenced: the argument checks come first
    box = np.array([6.0, 4.9, 6.0], np.float32)  # 2.5 > 4.9 / 2
    rc = lib.b2md_forces_noalloc(dummy, 100, box.ctypes.data_as(ctypes.c_void_p), 1,
                                 params.ctypes.data_as(ctypes.c_void_p), 0, dummy, dummy, None)
    assert rc == capi.B2MD_ERR_ARG
    assert b"half" in lib.b2md_last_error()
