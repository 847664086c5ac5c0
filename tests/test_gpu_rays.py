"""GPU ray bundles (mpf_rays_propagate, Integrator::propagate) against the
reference's outputs (tests/golden/rays.npz) and the C oracle.

Tolerances: exact mode is bit-identical (sizes and every column of the central
trajectory, the angular diameter distance included).  Fast mode (FP32
gathers): same accept / reject decisions and sizes within 1 point; positions
within 1e-9 and redshift within 1e-7 relative, the distance within 1e-5
relative (it is a difference of nearby rays' positions)."""
import numpy as np
import pytest

from conftest import load_golden
from test_rays_oracle import central_photons

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rays_dev(gpu_lib, pkg):
    g = load_golden("rays")
    tree = pkg.Octree.from_records(g["records"])
    cos = pkg.Cosmology(g["cosmo_t"], g["cosmo_a"], g["cosmo_dadt"], g["cosmo_d2adt2"])
    yield g, tree, cos
    tree.close()
    cos.close()


def _run(pkg, g, tree, cos, i, order, exact, cap=400):
    ph = central_photons(g)[i:i + 1]
    return pkg.rays_propagate(tree, cos, ph, float(g["cosmo_length"]), int(g["count"][i]), float(g["angle"][i]),
                              rotation=g["rotation"][i:i + 1], interpolation=str(g["interp"][i]), amin=float(g["amin"][i]),
                              nsteps=int(g["nsteps"]), order=order, exact=exact, capacity=cap)


@pytest.mark.parametrize("order", [1, 2])
def test_bundles_exact_bit_exact(rays_dev, pkg, order):
    g, tree, cos = rays_dev
    sizes, ref = g["ref_sizes_o%d" % order], g["ref_traj_o%d" % order]
    for i in range(sizes.shape[0]):
        s, t = _run(pkg, g, tree, cos, i, order, True)
        assert s[0] == sizes[i], i
        np.testing.assert_array_equal(t[0, :sizes[i]].view(np.uint64), ref[i, :sizes[i]].view(np.uint64))


@pytest.mark.parametrize("order", [1, 2])
def test_bundles_fast_within_tolerance(rays_dev, pkg, order):
    g, tree, cos = rays_dev
    sizes, ref = g["ref_sizes_o%d" % order], g["ref_traj_o%d" % order]
    for i in range(sizes.shape[0]):
        s, t = _run(pkg, g, tree, cos, i, order, False)
        assert (s[0] == 0) == (sizes[i] == 0), i
        if sizes[i] == 0:
            continue
        assert abs(int(s[0]) - int(sizes[i])) <= 1
        m = min(int(s[0]), int(sizes[i])) - 1
        got, want = t[0, :m], ref[i, :m]
        assert np.all(np.abs(got[:, 3:6] - want[:, 3:6]) <= 1e-9)
        assert np.all(np.abs(got[:, 19] - want[:, 19]) <= 1e-7 * np.abs(want[:, 19]) + 1e-12)
        assert np.all(np.abs(got[:, 22] - want[:, 22]) <= 1e-5 * np.abs(want[:, 22]) + 1e-30)


@pytest.mark.parametrize("order", [1, 2])
def test_bundles_fast_records_every_column(rays_dev, pkg, order):
    """Every directly stored column of a fast trajectory against the exact
    mode's.  A fast gather is good to 2e-6 of the field's scale and the state to
    better, so a column agrees to 1e-5 of its largest value, and the two running
    sums to 1e-5 of the sum of their terms at the field's largest values: isw of
    2 |dphidt| dt / c^2, iswold of (2 |grad phi| dx length + 2 |phi|) / c^2.  A
    sum that the exact mode reports is never all zero."""
    g, tree, cos = rays_dev
    c2 = 299792458.0 ** 2
    length = float(g["cosmo_length"])
    seen = 0
    for i in range(g["ref_sizes_o%d" % order].shape[0]):
        se, te = _run(pkg, g, tree, cos, i, order, True)
        sf, tf = _run(pkg, g, tree, cos, i, order, False)
        m = int(min(se[0], sf[0])) - 1
        if m < 2:
            continue
        e, f = te[0, :m], tf[0, :m]
        for col in (1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 19, 22, 25, 26, 27, 28):
            assert np.abs(f[:, col] - e[:, col]).max() <= 1e-5 * np.abs(e[:, col]).max() + 1e-30, (i, col)
        units = {23: 2 * np.abs(e[:, 27]).max() * np.abs(np.diff(e[:, 2])).sum() / c2,
                 24: (2 * np.abs(e[:, 14:17]).max() * np.abs(np.diff(e[:, 3:6], axis=0)).sum() * length +
                      2 * np.abs(e[:, 13]).max()) / c2}
        for col, unit in units.items():
            assert np.abs(f[:, col] - e[:, col]).max() <= 1e-5 * unit, (i, col)
            assert f[:, col].any() == e[:, col].any(), (i, col)
            seen += int(e[:, col].any())
    assert seen


def test_batch_of_bundles_matches_oracle(rays_dev, pkg, oracle_mod, synth):
    """Many bundles in one call (the trajectory buffers hold all of them at
    once) against the C oracle, exact mode."""
    g, tree, cos = rays_dev
    n = 24
    grid = synth.photon_grid(5, 1.0, 1.0)[:n]
    ph = np.concatenate([grid[:, :3], grid[:, 3:]], axis=1)
    rot = np.linspace(0.0, 3.0, n)
    kw = dict(nsteps=int(g["nsteps"]), order=2)
    sizes, traj = pkg.rays_propagate(tree, cos, ph, float(g["cosmo_length"]), 6, np.radians(0.25), rotation=rot,
                                     interpolation="r", exact=True, capacity=400, **kw)
    O = oracle_mod.Oracle(g["records"], {"t": g["cosmo_t"], "a": g["cosmo_a"], "dadt": g["cosmo_dadt"]},
                          float(g["cosmo_length"]), nthreads=1)
    for i in range(n):
        ref = O.propagate_bundle(ph[i], 6, np.radians(0.25), rot[i], "r", 0.0, **kw)
        assert sizes[i] == ref.shape[0], i
        np.testing.assert_array_equal(traj[i, :sizes[i]].view(np.uint64), ref.view(np.uint64))
    assert (sizes > 0).sum() >= n // 2


@pytest.mark.parametrize("capacity", [400, 1500])
def test_central_points_come_back_over_several_copies(rays_dev, pkg, oracle_mod, synth, capacity):
    """More points than one copy of the results holds, rejected bundles among
    them: bundles over the whole batch against the C oracle, exact mode, and
    nothing written behind a trajectory's end."""
    g, tree, cos = rays_dev
    n = 200
    ph = np.resize(synth.photon_grid(15, 1.0, 1.0), (n, 6)).copy()
    ph[1::7, 0] = 0.4                                    # leaves the box too soon: rejected
    rot = np.linspace(0.0, 3.0, n)
    kw = dict(nsteps=int(g["nsteps"]), order=1)
    sizes, traj = pkg.rays_propagate(tree, cos, ph, float(g["cosmo_length"]), 2, np.radians(0.25), rotation=rot,
                                     interpolation="r", exact=True, capacity=capacity, **kw)
    assert sizes.max() * n * traj.shape[2] * 8 > 4 << 20 and (sizes == 0).any()
    O = oracle_mod.Oracle(g["records"], {"t": g["cosmo_t"], "a": g["cosmo_a"], "dadt": g["cosmo_dadt"]},
                          float(g["cosmo_length"]), nthreads=1)
    for i in list(range(0, n, 17)) + [1, 8, n - 1]:
        ref = O.propagate_bundle(ph[i], 2, np.radians(0.25), rot[i], "r", 0.0, **kw)
        assert sizes[i] == ref.shape[0], i
        np.testing.assert_array_equal(traj[i, :sizes[i]].view(np.uint64), ref.view(np.uint64))
    for i in range(n):
        assert not traj[i, sizes[i]:].any(), i


def test_capacity_too_small_is_an_error(rays_dev, pkg):
    g, tree, cos = rays_dev
    with pytest.raises(pkg.MpfError):
        _run(pkg, g, tree, cos, 0, 2, True, cap=10)


def test_flrw_reference_bundle_bit_exact(rays_dev, pkg):
    """The rays driver's FLRW reference bundle (Order = -1 on a uniform octree)
    against the reference's own, every 8th point and the last."""
    g, tree, cos = rays_dev
    level, nst, every = int(g["flrw_level"]), int(g["flrw_nsteps"]), int(g["flrw_every"])
    ph = np.array([[0.0, 0.0, 0.0, 1.0, 0.0, 0.0]])     # Integrator::launch(0, 0, 0, 2, 0, 0)
    for j in range(g["flrw_count"].shape[0]):
        size = int(g["flrw_size_%d" % j])
        sizes, traj = pkg.rays_propagate(tree, cos, ph, float(g["cosmo_length"]), int(g["flrw_count"][j]),
                                         float(g["flrw_angle"][j]), interpolation=str(g["flrw_interp"][j]), nsteps=nst,
                                         order=1, exact=True, capacity=size + 8, homogeneous_level=level)
        assert sizes[0] == size
        np.testing.assert_array_equal(traj[0, :size:every].view(np.uint64), g["flrw_traj_%d" % j].view(np.uint64))
        np.testing.assert_array_equal(traj[0, size - 1].view(np.uint64), g["flrw_last_%d" % j].view(np.uint64))
