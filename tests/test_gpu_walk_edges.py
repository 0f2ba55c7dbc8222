"""Inputs, limits and call forms at which the FP64 walks, their scratch and the
dispatch between them can go wrong."""
import numpy as np
import pytest

import slsimlib_b200 as glb
from slsimlib_b200 import synth

pytestmark = pytest.mark.gpu


def _cluster(seed, n, size=0.01):
    r = np.random.default_rng(seed)
    p = np.zeros(n, dtype=synth.PARTICLE_DTYPE)
    p["x"] = np.concatenate([r.normal(0, 0.1, (n - n // 3, 3)), r.uniform(-1, 1, (n // 3, 3))])[:n]
    p["Mass"] = r.uniform(0.5, 2.0, n)
    p["Size"] = size * 10 ** r.uniform(-1, 1, n)
    return p


def _device_force(t, x, precision=glb.PREC_FP64, stream=None):
    import torch
    d = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    o = torch.full((len(x), 5), np.nan, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    t.force_device(len(x), d.data_ptr(), o.data_ptr(), precision, stream)
    torch.cuda.synchronize()
    return o.cpu().numpy()


class alloc_limit:
    """Device allocations of this thread above `nbytes` are refused inside the block."""

    def __init__(self, nbytes):
        self.nbytes = nbytes

    def __enter__(self):
        assert glb.load_library().glb_set_option(2, self.nbytes) == 0

    def __exit__(self, *a):
        glb.load_library().glb_set_option(2, 0)


def _refused(f):
    with pytest.raises(glb.GlamerError) as e:
        f()
    assert "out of memory" in str(e.value)


def _recur(t, x):
    a, k, g, ph = t.force2D_recur(x)
    return np.concatenate([a, k[:, None], g[:, :2], ph[:, None]], axis=1)


# NaNs of either sign whose low words, read as table indices, lie far outside any table.
NAN_BITS = np.array([0xFFFFFFFFE0000000, 0xFFF8000000000000, 0xFFFFFFFFFFFFFFFF, 0xFFF800007FFFFFFF, 0x7FF8000080000000,
                     0xFFF0000000100000], dtype=np.uint64)


@pytest.mark.parametrize("n", [64, 1 << 16])
@pytest.mark.parametrize("kw", [dict(inv_screening_scale=1.0), dict(inv_screening_scale=2.0, inv_area=0.1)])
def test_nan_payloads_stay_inside_the_tables(n, kw):
    t = glb.TreeQuadParticles(_cluster(1, 5000), bucket=5, theta_force=0.1, **kw)
    x = np.random.default_rng(2).normal(0, 0.3, (n, 2))
    y = x.copy()
    bad = np.arange(3, n, 41)
    y[bad, 0] = np.resize(NAN_BITS, len(bad)).view(np.float64)
    y[bad[::2], 1] = y[bad[::2], 0]
    ok = np.setdiff1d(np.arange(n), bad)
    for f in (_device_force, _recur):
        a, b = f(t, x), f(t, y)
        assert np.array_equal(a[ok], b[ok])
        assert np.all(np.isnan(b[bad][:, [0, 1, 3, 4]]))


def test_nan_payloads_in_lenses_and_served_requests():
    spec = synth.light_cone(seed=5, n_total=30000, n_planes=2, halos_per_plane=4)
    lens = glb.lens_from_spec(spec)
    for n in (97, 1 << 16, 131072):  # shared walks, one and two rays per lane
        x = np.random.default_rng(3).normal(0, 10 * synth.ARCSEC, (n, 2))
        y = x.copy()
        bad = np.arange(5, n, 29)
        y[bad, 1] = np.resize(NAN_BITS, len(bad)).view(np.float64)
        ok = np.setdiff1d(np.arange(n), bad)
        (y0, A0), (y1, A1) = lens.rayshooterInternal(x), lens.rayshooterInternal(y)
        assert np.array_equal(y0[ok], y1[ok]) and np.array_equal(A0[ok], A1[ok])
        assert np.all(np.isnan(A1[bad]).any(axis=1))
        if n == 97:
            srv = glb.Server([lens], precision=glb.PREC_FP64)
            got = [srv.wait(srv.submit(0, r))[:2] for r in (x, y)]
            srv.close()
            assert np.array_equal(got[0][0][ok], got[1][0][ok]) and np.array_equal(got[0][1][ok], got[1][1][ok])
            assert np.all(np.isnan(got[1][1][bad]).any(axis=1))


def _lens(n=20000, planes=2):
    return glb.lens_from_spec(synth.light_cone(seed=6, n_total=n, n_planes=planes, halos_per_plane=4))


@pytest.mark.parametrize("limit", [1 << 20, 80 * 60000])  # the call's staging, the workspace behind it
@pytest.mark.parametrize("precision", [glb.PREC_FP64, glb.PREC_SPLIT])
def test_lens_calls_after_a_refused_allocation(limit, precision):
    lens = _lens()
    x = np.random.default_rng(1).normal(0, 10 * synth.ARCSEC, (60000, 2))
    zs = np.full(len(x), 2.0)
    want = lens.rayshooterInternal(x[:3000], None, precision)
    grid = glb.GridMap(lens, 48, (0.0, 0.0), 20 * synth.ARCSEC, precision).y
    for again in range(2):
        with alloc_limit(limit):
            _refused(lambda: lens.rayshooterInternal(x, None, precision))
            _refused(lambda: lens.rayshooterInternal(x, zs, precision))
            _refused(lambda: glb.GridMap(lens, 300, (0.0, 0.0), 20 * synth.ARCSEC, precision))
        for got, ref in zip(lens.rayshooterInternal(x[:3000], None, precision), want):
            assert np.array_equal(got, ref)
        assert np.array_equal(glb.GridMap(lens, 48, (0.0, 0.0), 20 * synth.ARCSEC, precision).y, grid)


def test_trees_and_smoothing_after_a_refused_allocation():
    p = _cluster(2, 40000)
    x = np.random.default_rng(4).normal(0, 0.3, (50000, 2))
    t = glb.TreeQuadParticles(p, bucket=5, theta_force=0.3)
    want = _recur(t, x[:2000])
    small, size = p[:3000].copy(), p.copy()
    glb.calculate_smoothing(16, small)
    with alloc_limit(1 << 19):
        _refused(lambda: glb.TreeQuadParticles(p, bucket=5, theta_force=0.3))
        _refused(lambda: _recur(t, x))
        _refused(lambda: glb.calculate_smoothing(16, size))
    again = p[:3000].copy()
    glb.calculate_smoothing(16, again)
    assert np.array_equal(small["Size"], again["Size"])
    assert np.array_equal(_recur(t, x[:2000]), want)
    u = glb.TreeQuadParticles(p, bucket=5, theta_force=0.3)
    assert np.array_equal(_recur(u, x[:2000]), want)


def _noalloc(lens, x):
    import torch
    d = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    y = torch.empty((len(x), 2), dtype=torch.float64, device="cuda")
    A = torch.empty((len(x), 4), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    glb._check(glb.load_library().glb_lens_rayshoot_noalloc(lens._h, len(x), d.data_ptr(), None, y.data_ptr(),
                                                            A.data_ptr(), glb.PREC_FP64, None))
    torch.cuda.synchronize()
    return y.cpu().numpy(), A.cpu().numpy()


@pytest.mark.parametrize("n", [1, 700, 4097])
def test_walks_are_not_shared_without_memory_for_it(n):
    """The sums of shared walks take up to 100 MB; a call that cannot have them
    gives the results of one warp per 32 rays, which needs none."""
    limit = {1: 1 << 14}.get(n, 1 << 20)
    lens, p = _lens(200000), _cluster(4, 60000)
    x = np.random.default_rng(5).normal(0, 10 * synth.ARCSEC, (n, 2))
    want = _noalloc(lens, x)
    t, u = (glb.TreeQuadParticles(p, bucket=5, theta_force=0.1) for _ in range(2))
    r = np.random.default_rng(6).normal(0, 0.3, (1 << 16, 2))
    whole, few, host = _device_force(t, r)[:n], _device_force(t, r[:n]), _recur(t, r[:n])
    assert n == 1 or not np.array_equal(few, whole)  # shared: another order of the sum
    with alloc_limit(limit):
        for again in range(2):
            got = lens.rayshooterInternal(x)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
            assert np.array_equal(_device_force(u, r[:n]), whole)
            assert np.abs(_recur(u, r[:n]) - host).max() <= 1e-11 * np.abs(host).max()
    shared = lens.rayshooterInternal(x)
    assert n == 1 or not np.array_equal(shared[1], want[1])


def test_host_forces_in_smaller_pieces_where_memory_is_refused():
    t = glb.TreeQuadParticles(_cluster(7, 3000), bucket=20, theta_force=0.3)
    x = np.random.default_rng(8).normal(0, 0.3, (300001, 2))
    want = _recur(t, x)
    u = glb.TreeQuadParticles(_cluster(7, 3000), bucket=20, theta_force=0.3)
    with alloc_limit(110 * 100000):
        got = _recur(u, x)
    assert np.abs(got - want).max() <= 1e-11 * np.abs(want).max()


def test_device_forces_on_two_streams_overlap():
    """Small FP64 device calls on two streams use scratch of their own: a call
    on the second stream ends while the first still has work queued."""
    import torch
    t = glb.TreeQuadParticles(_cluster(9, 200000), bucket=5, theta_force=0.05)
    x = np.random.default_rng(10).normal(0, 0.3, (20000, 2))
    want, few = _device_force(t, x), _device_force(t, x[:64])
    d = torch.from_numpy(x).cuda()
    out = torch.zeros((40, len(x), 5), dtype=torch.float64, device="cuda")
    small = torch.zeros((64, 5), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for o in out:
        t.force_device(len(x), d.data_ptr(), o.data_ptr(), glb.PREC_FP64, a.cuda_stream)
    t.force_device(64, d.data_ptr(), small.data_ptr(), glb.PREC_FP64, b.cuda_stream)
    b.synchronize()
    assert not a.query()
    assert np.array_equal(small.cpu().numpy(), few)
    a.synchronize()
    assert all(np.array_equal(o, want) for o in out.cpu().numpy())


def test_device_forces_of_several_threads_and_sizes():
    import threading
    import torch
    t = glb.TreeQuadParticles(_cluster(11, 50000), bucket=5, theta_force=0.1)
    x = np.random.default_rng(12).normal(0, 0.3, (5000, 2))
    sizes = (17, 5000, 500, 4999, 33, 2500)
    want = {n: _device_force(t, x[:n]) for n in sizes}
    d = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        torch.cuda.set_device(0)
        s = torch.cuda.Stream()
        for n in sizes[k:] + sizes[:k]:
            o = torch.zeros((n, 5), dtype=torch.float64, device="cuda")
            torch.cuda.current_stream().synchronize()
            t.force_device(n, d.data_ptr(), o.data_ptr(), glb.PREC_FP64, s.cuda_stream)
            s.synchronize()
            if not np.array_equal(o.cpu().numpy(), want[n]):
                wrong.append(n)

    th = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for q in th:
        q.start()
    for q in th:
        q.join()
    assert not wrong


def test_a_captured_device_force_is_one_unshared_launch():
    import torch
    t = glb.TreeQuadParticles(_cluster(13, 60000), bucket=5, theta_force=0.1)
    x = np.random.default_rng(14).normal(0, 0.3, (1 << 16, 2))
    want = _device_force(t, x)[:300]
    d = torch.from_numpy(x[:300].copy()).cuda()
    o = torch.zeros((300, 5), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        t.force_device(300, d.data_ptr(), o.data_ptr(), glb.PREC_FP64, s.cuda_stream)
    for again in range(2):
        o.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(o.cpu().numpy(), want)


def test_growing_and_shrinking_lens_calls():
    lens, other = _lens(), _lens()
    x = np.random.default_rng(15).normal(0, 10 * synth.ARCSEC, (6000, 2))
    for n in (500, 6000, 40, 3000, 5999, 1):
        got, want = lens.rayshooterInternal(x[:n]), other.rayshooterInternal(x[:n])
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


def test_host_forces_of_two_callers_and_many_sizes():
    import threading
    t = glb.TreeQuadParticles(_cluster(16, 30000), bucket=5, theta_force=0.3)
    x = np.random.default_rng(17).normal(0, 0.3, (20000, 2))
    sizes = (1, 20000, 700, 4097, 64)
    want = {n: _recur(t, x[:n]) for n in sizes}
    wrong = []

    def work(k):
        for n in sizes[k:] + sizes[:k]:
            if not np.array_equal(_recur(t, x[:n]), want[n]):
                wrong.append(n)

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for q in th:
        q.start()
    for q in th:
        q.join()
    assert not wrong


def test_repeated_host_forces_keep_no_more_memory():
    """The workspace of a host call (100 MB here) is not mapped and unmapped by
    each: what the device has free does not change from call to call."""
    import torch
    t = glb.TreeQuadParticles(_cluster(18, 200000), bucket=5, theta_force=0.1)
    x = np.random.default_rng(19).normal(0, 0.3, (5000, 2))
    _recur(t, x)
    free = torch.cuda.mem_get_info()[0]
    for n in (3000, 5000, 400, 4999):
        _recur(t, x[:n])
        assert torch.cuda.mem_get_info()[0] == free


def test_a_refused_allocation_takes_back_the_unused_scratch():
    import torch
    t = glb.TreeQuadParticles(_cluster(20, 200000), bucket=5, theta_force=0.1)
    x = np.random.default_rng(21).normal(0, 0.3, (3000, 2))
    want = _recur(t, x)
    lens = _lens()
    lens.rayshooterInternal(np.zeros((1, 2)))
    free = torch.cuda.mem_get_info()[0]
    with alloc_limit(1 << 20):
        _refused(lambda: lens.rayshooterInternal(np.zeros((60000, 2))))
    assert torch.cuda.mem_get_info()[0] >= free + (64 << 20)
    assert np.array_equal(_recur(t, x), want)


@pytest.mark.parametrize("n,bucket,theta,limit", [
    (20000, 5, 0.1, 1 << 20), (20000, 20, 0.3, 1 << 20), (60000, 20, 0.1, 1 << 20),  # by strips from there on
    (60000, 20, 0.2, 1 << 18), (600000, 20, 0.1, 1 << 18),                            # node by node
    (60000, 5, 0.1, 1 << 16), (20000, 5, 0.3, 1 << 16), (60000, 20, 0.3, 1 << 16),
])
def test_device_forces_on_both_sides_of_their_limit(n, bucket, theta, limit):
    t = glb.TreeQuadParticles(_cluster(n + bucket, n), bucket=bucket, theta_force=theta, inv_screening_scale=1.0)
    x = np.random.default_rng(22).normal(0, 0.3, (limit, 2))
    few = _device_force(t, x[:3000])
    assert np.array_equal(_device_force(t, x[:2999]), few[:2999])
    for m in (limit - 1, limit):
        got = _device_force(t, x[:m])
        assert np.all(np.isfinite(got))
        assert np.all(np.abs(got[:3000] - few).max(axis=0) <= 1e-11 * np.abs(few).max(axis=0))


@pytest.mark.parametrize("n", [1, 100, 70000])
def test_periodic_device_forces(n):
    t = glb.TreeQuadParticles(_cluster(23, 900), bucket=5, theta_force=0.1, periodic_buffer=True,
                              inv_screening_scale=1.0)
    x = np.random.default_rng(24).normal(0, 0.3, (n, 2))
    want = _recur(t, x)[:, :5]
    assert np.all(np.abs(_device_force(t, x) - want).max(axis=0) <= 1e-11 * np.abs(want).max(axis=0))


def test_lens_calls_with_fewer_rays_than_nodes():
    """One plane of 100,000 nodes: calls on both sides of that many rays share
    and do not share their walks, and agree."""
    p = _cluster(25, 700000, 0.001)
    p["Mass"] *= 1e9
    lens = glb.Lens(2.0)
    lens.insertMainHalo(glb.LensHaloParticles(p, 0.3), True)
    x = np.random.default_rng(26).normal(0, 60 * synth.ARCSEC, (130000, 2))
    zs = np.random.default_rng(27).uniform(0.1, 3.0, len(x))
    for z in (None, zs):
        want = lens.rayshooterInternal(x[:65535], None if z is None else z[:65535])
        for n in (65536, 80000, 130000):
            y, A = lens.rayshooterInternal(x[:n], None if z is None else z[:n])
            assert np.abs(y[:65535] - want[0]).max() < 1e-11 * np.abs(want[0]).max()
            assert np.abs(A[:65535] - want[1]).max() < 1e-8 * np.abs(want[1]).max()
            got = _noalloc(lens, x[:n]) if n <= 65536 and z is None else (y, A)
            assert np.abs(got[0] - y).max() < 1e-11 * np.abs(y).max()


@pytest.mark.parametrize("n,bucket,theta,kw,limit", [
    (20000, 5, 0.1, {}, 1 << 18), (600000, 5, 0.1, {}, 1 << 17), (20000, 20, 0.3, dict(inv_area=0.1), 1 << 18),
    (60000, 20, 0.2, dict(inv_area=0.1), 1 << 17), (60000, 5, 0.3, dict(inv_screening_scale=1.0, inv_area=0.2), 1 << 16),
])
def test_host_forces_on_both_sides_of_their_limit(n, bucket, theta, kw, limit):
    t = glb.TreeQuadParticles(_cluster(n + bucket, n), bucket=bucket, theta_force=theta, **kw)
    x = np.random.default_rng(28).normal(0, 0.3, (limit, 2))
    few = _recur(t, x[:3000])
    for m in (limit - 1, limit):
        got = _recur(t, x[:m])
        assert np.all(np.isfinite(got))
        assert np.all(np.abs(got[:3000] - few).max(axis=0) <= 1e-11 * np.abs(few).max(axis=0))
    assert np.all(np.abs(_device_force(t, x[:3000]) - few[:, :5]).max(axis=0) <= 1e-11 * np.abs(few[:, :5]).max(axis=0))


@pytest.mark.parametrize("np_,theta", [(700, 0.1), (30000, 0.3)])
def test_node_by_node_potential_matches_the_oracle(np_, theta):
    from tests import harness as H
    from tests.test_gpu_parity import force_err, pack
    p = _cluster(np_, np_, 0.02)
    x = np.random.default_rng(29).normal(0, 0.3, (70000, 2))
    x[0] = p["x"][0, :2]
    for periodic in (False, True):
        if periodic and np_ > 1000:
            continue
        t = glb.TreeQuadParticles(p, bucket=5, theta_force=theta, inv_screening_scale=1.0, periodic_buffer=periodic)
        o = H.OracleTree(p, bucket=5, theta=theta, inv_area=0.0, inv_screening=1.0, periodic=int(periodic))
        got = pack(*t.force2D_recur(x))[:257]
        err, cols = force_err(got, o.force(x[:257]))
        assert err < 1e-9, cols


@pytest.mark.parametrize("sides", [(33,), (300, 300)])  # the list walk, and too many rays for it
def test_split_batches_of_a_large_tree(sides):
    """A tree of about 130,000 nodes in a split-form batch: every ray's result is
    the lens path's of a plane with two particle haloes (a walk per ray)."""
    p, q = _cluster(30, 900000, 0.001), _cluster(31, 40, 0.05)
    for c in (p, q):
        c["Mass"] *= 1e9
    lens = glb.Lens(2.0)
    for c in (p, q):
        lens.insertMainHalo(glb.LensHaloParticles(c, 0.3), True)
    rng = 100 * synth.ARCSEC
    b = glb.GridBatch([lens] * len(sides), sides, [(0.0, 0.0)] * len(sides), [rng] * len(sides), glb.PREC_SPLIT)
    b.run()
    for i, side in enumerate(sides):
        y, A = b.result(i)
        g = glb.GridMap(lens, side, (0.0, 0.0), rng, glb.PREC_SPLIT)
        assert np.abs(y - g.y).max() <= 1e-13 * np.abs(g.y).max()
        assert np.abs(A - g.A).max() <= 1e-13 * np.abs(g.A).max()


def _mixed_lenses():
    plain = [_lens(30000, 2), _lens(20000, 1)]
    spec = synth.light_cone(seed=9, n_total=25000, n_planes=2, halos_per_plane=4)
    spec.halos.append(synth.NFWHalo(3e13, 0.4, 0.7, 6.0))
    return plain, glb.lens_from_spec(spec)


@pytest.mark.parametrize("block", [64, 128, 256])
@pytest.mark.parametrize("graph", [False, True])
def test_batched_lenses_do_not_depend_on_each_other(block, graph):
    """FP64 batches: lenses with and without NFW haloes in one batch have the bits
    that they have in batches of their own; those without, the lens path's terms."""
    plain, nfw = _mixed_lenses()
    order = [plain[0], nfw, plain[1], nfw]
    sides, rng = [33, 20, 64, 7], 40 * synth.ARCSEC
    b = glb.GridBatch(order, sides, [(0.0, 0.0)] * 4, [rng] * 4, glb.PREC_FP64)
    b.set_block(block)
    b.run(graph)
    for i, (lens, side) in enumerate(zip(order, sides)):
        one = glb.GridBatch([lens], [side], [(0.0, 0.0)], [rng], glb.PREC_FP64)
        one.run(False)
        (y, A), (y1, A1) = b.result(i), one.result(0)
        assert np.array_equal(y, y1) and np.array_equal(A, A1)
        g = glb.GridMap(lens, side, (0.0, 0.0), rng, glb.PREC_FP64)
        assert np.abs(y - g.y).max() <= 1e-11 * np.abs(g.y).max()
        if lens is not nfw:
            assert np.abs(A - g.A).max() <= 1e-8 * np.abs(g.A).max()


def test_served_models_do_not_depend_on_each_other():
    plain, nfw = _mixed_lenses()
    x = np.random.default_rng(32).normal(0, 10 * synth.ARCSEC, (500, 2))
    both = glb.Server([plain[0], nfw, plain[1]], precision=glb.PREC_FP64)
    tickets = [both.submit(k, x[: 500 - 7 * k], 2.0) for k in (2, 1, 0, 1, 2)]
    got = [both.wait(t)[:2] for t in tickets]
    both.close()
    for k, (y, A) in zip((2, 1, 0, 1, 2), got):
        own = glb.Server([[plain[0], nfw, plain[1]][k]], precision=glb.PREC_FP64)
        y1, A1 = own.wait(own.submit(0, x[: 500 - 7 * k], 2.0))[:2]
        own.close()
        assert np.array_equal(y, y1) and np.array_equal(A, A1)


def test_small_calls_after_builds_map_no_memory():
    """Trees built and freed leave their pool in pieces; the scratch of a small
    call is not mapped and given back by each call for that."""
    import torch
    lens = _lens(400000)
    x = np.random.default_rng(33).normal(0, 10 * synth.ARCSEC, (4097, 2))
    for n in (50000, 300000, 150000):
        glb.TreeQuadParticles(_cluster(n, n), bucket=5, theta_force=0.1)
    want = lens.rayshooterInternal(x)
    free = torch.cuda.mem_get_info()[0]
    for again in range(3):
        got = lens.rayshooterInternal(x)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        assert torch.cuda.mem_get_info()[0] == free


@pytest.mark.parametrize("bucket", [5, 20])
def test_builds_without_their_scratch_in_one_piece(bucket):
    """Where the one piece (over 240 bytes a particle) cannot be had, a build goes on
    with the buffers' own allocations."""
    p = _cluster(34, 100000)
    x = np.random.default_rng(35).normal(0, 0.3, (500, 2))
    want = _recur(glb.TreeQuadParticles(p, bucket=bucket, theta_force=0.1), x)
    with alloc_limit((1 << 20) + 240 * len(p)):
        t = glb.TreeQuadParticles(p, bucket=bucket, theta_force=0.1)
    assert np.array_equal(_recur(t, x), want)


@pytest.mark.parametrize("n", [16384, 32768, 32769, 36000, 65536, 65537])
def test_trees_at_the_edges_of_their_allocations(n):
    """Particles and nodes lie in one allocation or two (1 MB): forces of every form
    against the oracle (the split form's within its 1e-5 at the 99.9th percentile)."""
    from tests import harness as H
    from tests.test_gpu_parity import force_err, pack, vec_err
    p = _cluster(n, n, 0.002)
    x = np.random.default_rng(36).normal(0, 0.3, (1000, 2))
    t = glb.TreeQuadParticles(p, bucket=20, theta_force=0.1, inv_screening_scale=1.0)
    want = H.OracleTree(p, bucket=20, theta=0.1, inv_area=0.0, inv_screening=1.0, periodic=0).force(x[:100])
    assert force_err(pack(*t.force2D_recur(x[:100])), want)[0] < 1e-9
    fp64, split = _device_force(t, x), _device_force(t, x, glb.PREC_SPLIT)
    assert np.quantile(vec_err(split[:, :2], fp64[:, :2]), 0.999) < 1e-5


def _signed(seed, n, size):
    p = _cluster(seed, n, size)
    p["Mass"] *= np.where(np.random.default_rng(seed + 100).random(n) < 0.3, -1e9, 1e9).astype(np.float32)
    return p


@pytest.mark.parametrize("n", [200, 70000, 131072])
def test_two_particle_haloes_on_one_plane(n):
    """FP64 planes with two particle haloes (the kernel without a tree in its
    parameters) against the oracle."""
    from tests import harness as H
    spec = synth.LensSpec(zsource=2.0, halos=[
        synth.ParticlePlane(_signed(40, 3000, 0.02), 0.3, inv_area=0.0), synth.ParticlePlane(_cluster(41, 500, 0.05), 0.3),
        synth.ParticlePlane(_signed(42, 2000, 0.01), 0.7)])
    lens = glb.lens_from_spec(spec)
    assert lens.getNplanes() == 2
    x = np.random.default_rng(43).normal(0, 30 * synth.ARCSEC, (n, 2))
    y, A = lens.rayshooterInternal(x)
    yo, Ao = H.OracleLens(spec).rayshoot(x[:200])
    assert np.abs(y[:200] - yo).max() < 1e-9 * np.abs(yo).max()
    assert np.abs(A[:200] - Ao).max() < 1e-8 * np.abs(Ao).max()


@pytest.mark.parametrize("inv_area", [0.0, 0.3])
@pytest.mark.parametrize("size", [0.001, 0.3])  # 0.3: most particles are softened at internal nodes
def test_two_rays_per_lane_with_sheets_signs_and_softening(inv_area, size):
    lens = glb.Lens(2.0)
    for z, s in ((0.3, 50), (0.8, 51)):
        lens.insertMainHalo(glb.LensHaloParticles(_signed(s, 8000, size), z, inv_area=inv_area), True)
    x = np.random.default_rng(52).normal(0, 40 * synth.ARCSEC, (131072, 2))
    zs = np.random.default_rng(53).uniform(0.05, 3.0, len(x))
    for z in (None, zs):
        y, A = lens.rayshooterInternal(x, z)  # two rays per lane
        assert np.all(np.isfinite(A))
        ys, As = lens.rayshooterInternal(x[:66049], None if z is None else z[:66049])  # one
        assert np.array_equal(y[:66049], ys) and np.array_equal(A[:66049], As)


@pytest.mark.parametrize("n", [100, 70001])
def test_two_large_particle_haloes_on_one_plane(n):
    """A tree of more than 2^18 nodes beside another on a plane: node by node, the
    terms of the two haloes on planes (nearly) of their own."""
    p, q = _cluster(60, 2000000, 0.0005), _cluster(61, 3000, 0.01)
    for c in (p, q):
        c["Mass"] *= 1e9
    x = np.random.default_rng(62).normal(0, 60 * synth.ARCSEC, (n, 2))
    both, one, two = glb.Lens(2.0), glb.Lens(2.0), glb.Lens(2.0)
    both.insertMainHalo(glb.LensHaloParticles(p, 0.3), True)
    both.insertMainHalo(glb.LensHaloParticles(q, 0.3), True)
    one.insertMainHalo(glb.LensHaloParticles(p, 0.3), True)
    two.insertMainHalo(glb.LensHaloParticles(q, 0.3), True)
    assert both.getNplanes() == 1
    (y, A), (y1, A1), (y2, A2) = (lens.rayshooterInternal(x) for lens in (both, one, two))
    # one plane: deflections and the Jacobian's deviations from unity add up
    assert np.abs(y - (y1 + y2 - x)).max() <= 1e-11 * np.abs(y).max()
    unit = np.array([1.0, 0.0, 0.0, 1.0])
    assert np.abs(A - (A1 + A2 - unit)).max() <= 1e-10 * np.abs(A).max()


def test_the_scratch_of_calls_at_once_is_kept():
    """Eight calls in flight on eight streams hold 80 MB each; the pool keeps them for
    the next eight instead of mapping memory for each call."""
    import torch
    t = glb.TreeQuadParticles(_cluster(63, 200000), bucket=5, theta_force=0.05)
    x = np.random.default_rng(64).normal(0, 0.3, (5000, 2))
    want = _device_force(t, x)
    lens = _lens()
    with alloc_limit(1 << 20):
        _refused(lambda: lens.rayshooterInternal(np.zeros((60000, 2))))  # gives back what the pools hold
    d = torch.from_numpy(x).cuda()
    out = torch.zeros((8, len(x), 5), dtype=torch.float64, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(8)]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for o, s in zip(out, streams):
        t.force_device(len(x), d.data_ptr(), o.data_ptr(), glb.PREC_FP64, s.cuda_stream)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] > 500 << 20
    assert all(np.array_equal(o, want) for o in out.cpu().numpy())
