"""The FP64 strip walk (csrc/walk_strip.cuh): one warp per 32 rays, and walks
shared by several warps in small calls, against the oracle's recursive walk and
against each other, at the edges of strips, warps and parts.

Tolerances: a walk adds at most a few thousand terms per component, each good
to a few 2^-53, so 1e-9 of the oracle (its own rounding and the cancellation of
terms included, as in test_gpu_parity) and 1e-11 between the two ways of
sharing (largest column value)."""
import numpy as np
import pytest

import slsimlib_b200 as glb
from slsimlib_b200 import synth
from tests import harness as H
from tests.test_gpu_parity import force_err, pack

pytestmark = pytest.mark.gpu


def _cluster(seed, n, size=0.01, sign=False):
    r = np.random.default_rng(seed)
    p = np.zeros(n, dtype=synth.PARTICLE_DTYPE)
    p["x"] = np.concatenate([r.normal(0, 0.1, (n - n // 3, 3)), r.uniform(-1, 1, (n // 3, 3))])[:n]
    p["Mass"] = r.uniform(0.5, 2.0, n) * (np.where(r.random(n) < 0.3, -1, 1) if sign else 1)
    p["Size"] = size * 10 ** r.uniform(-1, 1, n)
    return p


def _rays(seed, n):
    r = np.random.default_rng(seed)
    return r.normal(0, 0.3, (n, 2))


@pytest.mark.parametrize("np_,bucket,theta,kw", [
    (2, 1, 0.1, {}), (19, 5, 0.1, {}), (33, 1, 0.3, dict(inv_screening_scale=1.3)),
    (700, 1, 0.1, dict(inv_area=0.2)), (5000, 5, 0.1, dict(inv_screening_scale=2.0, inv_area=0.1)),
    (5000, 20, 0.0, {}), (3000, 40, 0.3, {}), (900, 5, 0.1, dict(periodic_buffer=True, inv_screening_scale=1.0)),
])
@pytest.mark.parametrize("n", [1, 31, 33, 65, 257])
def test_force_matches_oracle(np_, bucket, theta, kw, n):
    p = _cluster(np_ + bucket, np_, sign=np_ == 700)
    x = _rays(n, n)
    x[0] = p["x"][0, :2]  # on a particle
    t = glb.TreeQuadParticles(p, bucket=bucket, theta_force=theta, **kw)
    okw = dict(kw)
    o = H.OracleTree(p, bucket=bucket, theta=theta, inv_area=okw.get("inv_area", 0.0),
                     inv_screening=okw.get("inv_screening_scale", 0.0), periodic=int(okw.get("periodic_buffer", False)))
    err, cols = force_err(pack(*t.force2D_recur(x)), o.force(x))
    assert err < 1e-9, cols


def _device_force(t, x):
    import torch
    d = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    out = torch.empty((len(x), 5), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    t.force_device(len(x), d.data_ptr(), out.data_ptr(), glb.PREC_FP64)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("n", [1, 40, 4096, 4127])
def test_shared_and_single_walks_agree(n):
    p = _cluster(3, 60000)
    t = glb.TreeQuadParticles(p, bucket=5, theta_force=0.1, inv_screening_scale=1.0)
    x = _rays(8, 1 << 16)
    f = pack(*t.force2D_recur(x[:n]))  # shared walks, rays sorted
    g = _device_force(t, x)[:n]        # one warp per 32 rays, the caller's order
    h = _device_force(t, x[:n])        # shared walks, the caller's order
    for c in range(5):
        top = np.abs(g[:, c]).max()
        assert np.abs(f[:, c] - g[:, c]).max() <= 1e-11 * top and np.abs(h[:, c] - g[:, c]).max() <= 1e-11 * top


@pytest.mark.parametrize("n", [3000, 1 << 16])
def test_rays_do_not_depend_on_each_other(n):
    p = _cluster(5, 20000)
    t = glb.TreeQuadParticles(p, bucket=20, theta_force=0.1, inv_screening_scale=1.0)
    x = _rays(9, n)
    perm = np.random.default_rng(1).permutation(len(x))
    a, b = _device_force(t, x), _device_force(t, x[perm])
    assert np.array_equal(a[perm], b)
    f, g = pack(*t.force2D_recur(x)), pack(*t.force2D_recur(x[perm]))
    assert np.array_equal(f[perm], g)
    # rays that are not finite, or far away, leave the others alone
    y = x.copy()
    bad = np.arange(7, len(x), 97)
    y[bad[0::3]] = np.nan
    y[bad[1::3]] = np.inf
    y[bad[2::3]] = 1e9
    ok = np.setdiff1d(np.arange(len(x)), bad)
    assert np.array_equal(_device_force(t, y)[ok], a[ok])
    assert np.array_equal(pack(*t.force2D_recur(y))[ok], f[ok])
    h = _device_force(t, y)[bad]
    assert np.all(~np.isfinite(h[0::3, :2])) and np.all(np.isfinite(h[2::3]))


@pytest.mark.parametrize("n", [1, 63, 64, 2049])
def test_small_lens_calls_match_large_ones(n):
    spec = synth.light_cone(seed=11, n_total=60000, n_planes=3, halos_per_plane=4)
    lens = glb.lens_from_spec(spec)
    r = np.random.default_rng(2)
    x = r.normal(0, 10 * synth.ARCSEC, (1 << 16, 2))
    zs = r.uniform(0.05, 3.0, len(x))
    for z in (None, zs):
        y, A = lens.rayshooterInternal(x, z)
        ys, As = lens.rayshooterInternal(x[:n], None if z is None else z[:n])
        assert np.abs(ys - y[:n]).max() < 1e-11 * np.abs(y).max()
        assert np.abs(As - A[:n]).max() < 1e-8 * np.abs(A).max()


def test_two_rays_per_lane_match_one():
    """Grids whose ray counts take the two-ray kernel (131,044 rays: one wave of
    it) and the one-ray kernel (their first 66,049 rays) agree bit for bit."""
    spec = synth.light_cone(seed=12, n_total=40000, n_planes=2, halos_per_plane=4)
    lens = glb.lens_from_spec(spec)
    x = synth.grid_positions(362, range_rad=40 * synth.ARCSEC)
    y, A = lens.rayshooterInternal(x)
    ys, As = lens.rayshooterInternal(x[:66049])
    assert np.array_equal(y[:66049], ys) and np.array_equal(A[:66049], As)
    zs = np.random.default_rng(3).uniform(0.05, 3.0, len(x))
    y, A = lens.rayshooterInternal(x, zs)
    ys, As = lens.rayshooterInternal(x[:66049], zs[:66049])
    assert np.array_equal(y[:66049], ys) and np.array_equal(A[:66049], As)


@pytest.mark.parametrize("n,size,sign,inv_area", [
    (1, 0.01, False, 0.0), (2, 0.01, False, 0.0), (21, 0.5, False, 0.0), (700, 0.02, True, 0.3),
    (3000, 0.3, False, 0.2), (60000, 0.001, False, 0.0), (200000, 0.0005, False, 0.0),
    (3000000, 0.0002, False, 0.0),  # more nodes than the list walk takes
])
@pytest.mark.parametrize("side", [1, 5, 33, 96])
def test_list_walk_matches_the_walk_of_each_ray(n, size, sign, inv_area, side):
    """The batch's split form (list walk) against the lens path of a plane with
    two particle haloes (a walk per ray): the same FP32 blocks in the same
    order, so only the FP64 recursion may round differently."""
    p, q = _cluster(n + 1, n, size, sign), _cluster(n + 2, 40, 0.05)
    for c in (p, q):
        c["Mass"] *= 1e10
    lens = glb.Lens(2.0)
    lens.insertMainHalo(glb.LensHaloParticles(p, 0.3, inv_area=inv_area), True)
    lens.insertMainHalo(glb.LensHaloParticles(q, 0.3), True)
    assert lens.getNplanes() == 1
    rng = 100 * synth.ARCSEC
    b = glb.GridBatch([lens], [side], [(0.0, 0.0)], [rng], glb.PREC_SPLIT)
    for block in (64, 128, 256):
        b.set_block(block)
        b.run()
        y, A = b.result(0)
        g = glb.GridMap(lens, side, (0.0, 0.0), rng, glb.PREC_SPLIT)
        assert np.abs(y - g.y).max() <= 1e-13 * np.abs(g.y).max()
        assert np.abs(A - g.A).max() <= 1e-13 * np.abs(g.A).max()
