"""Launch shapes of the propagation kernels: a batch smaller than one full warp
per SM sub-partition runs with fewer rays a warp and, with the Jacobian, with
2, 3 or 6 lanes a ray.  A ray's result does not depend on the shape, so the
first n rays traced alone equal bit for bit the same rays of a batch that
runs full warps, on both sides of every change of shape."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu

# rays a warp = ceil(n / 608) on 152 SMs: 6 lanes a ray up to 5, 3 up to 10, 2 up to 16
SIZES = (1, 31, 608, 609, 3040, 3041, 6080, 6081, 9728, 9729, 19456)


@pytest.fixture(scope="module")
def rays(gpu_lib, pkg, synth):
    g = load_golden("amr")
    tree = pkg.Octree.from_records(g["records"])
    cos = pkg.Cosmology(g["cosmo_t"], g["cosmo_a"], g["cosmo_dadt"], g["cosmo_d2adt2"])
    launch = synth.photon_grid(200, 2.4, 2.4)
    yield tree, cos, float(g["cosmo_length"]), launch, {}
    tree.close()
    cos.close()


@pytest.mark.parametrize("order,jacobian", [(1, True), (2, True), (2, False)])
@pytest.mark.parametrize("n", SIZES)
def test_small_batches_equal_large_ones(rays, pkg, order, jacobian, n):
    tree, cos, length, launch, whole = rays
    kw = dict(nsteps=5, order=order, stop="redshift", stop_value=0.1, planes=np.array([0.04, 0.1]), jacobian=jacobian)
    if (order, jacobian) not in whole:
        whole[order, jacobian] = pkg.propagate(tree, cos, launch, length, **kw)
    s0, f0, p0, _ = whole[order, jacobian]
    s, f, p, rc = pkg.propagate(tree, cos, launch[:n], length, **kw)
    assert rc == 0
    np.testing.assert_array_equal(s, s0[:n])
    np.testing.assert_array_equal(f.view(np.uint64), f0[:n].view(np.uint64))
    np.testing.assert_array_equal(p.view(np.uint64), p0[:n].view(np.uint64))


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("n", (1, 609, 3041, 6081, 9729))
def test_small_exact_batches_equal_large_ones(rays, pkg, order, n):
    tree, cos, length, launch, whole = rays
    kw = dict(nsteps=4, order=order, stop="redshift", stop_value=0.03, planes=np.array([0.01, 0.03]), jacobian=True, exact=True)
    if ("exact", order) not in whole:
        whole["exact", order] = pkg.propagate(tree, cos, launch, length, **kw)
    s0, f0, p0, _ = whole["exact", order]
    s, f, p, rc = pkg.propagate(tree, cos, launch[:n], length, **kw)
    assert rc == 0
    np.testing.assert_array_equal(s, s0[:n])
    np.testing.assert_array_equal(f.view(np.uint64), f0[:n].view(np.uint64))
    np.testing.assert_array_equal(p.view(np.uint64), p0[:n].view(np.uint64))


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("n", (16383, 16384, 40000))
def test_ray_order_changes_no_ray(rays, pkg, order, n):
    """From 2^14 rays on a refined octree runs the rays in the order of their
    directions: any order of the caller's gives the same rays, directions in
    all eight octants and repeated ones among them."""
    tree, cos, length, launch, _ = rays
    rng = np.random.default_rng(n)
    some = launch[rng.permutation(launch.shape[0])[:n]].copy()
    some[::1000, 3:] = rng.normal(size=some[::1000, 3:].shape)
    some[1::1000] = some[0]
    kw = dict(nsteps=4, order=order, stop="redshift", stop_value=0.04, planes=np.array([0.04]), jacobian=True)
    s, f, p, _ = pkg.propagate(tree, cos, some, length, **kw)
    for lo in range(0, n, 8000):     # below the threshold: in the caller's order
        s0, f0, p0, _ = pkg.propagate(tree, cos, some[lo:lo + 8000], length, **kw)
        np.testing.assert_array_equal(s[lo:lo + 8000], s0)
        np.testing.assert_array_equal(f[lo:lo + 8000].view(np.uint64), f0.view(np.uint64))
        np.testing.assert_array_equal(p[lo:lo + 8000].view(np.uint64), p0.view(np.uint64))
