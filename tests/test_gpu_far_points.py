"""Points far outside the domain, at infinity and NaN, on an octree that fills
the domain (so that the wrapped and saturated integer coordinates find cells):
the exact gathers give the C oracle's bits, NaN where it gives NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FAR = [2.5, 5.99, 3e9, 2.0 ** 33, 2.0 ** 34, 2.0 ** 36, 1e12, 1e15, np.inf, -2.5, -1e12, -np.inf, np.nan]


@pytest.fixture(scope="module")
def full(synth):
    """All cells of levels 3 and 4."""
    rng = np.random.default_rng(4)
    recs = []
    for level in (3, 4):
        c = np.stack(np.meshgrid(*3 * [np.arange(2 ** level)], indexing="ij"), -1).reshape(-1, 3)
        r = np.zeros(c.shape[0], dtype=synth.RECORD)
        r["hi"], r["lo"] = synth.key_from_coords(level, c)
        for f in ("dphidt", "a", "dphidx", "dphidy", "dphidz", "phi", "rho"):
            r[f] = rng.uniform(0.5, 1.5, c.shape[0])
        recs.append(r)
    out = np.concatenate(recs)
    return out[np.lexsort((out["lo"], out["hi"]))]


@pytest.fixture(scope="module")
def oracle(full, oracle_mod):
    return oracle_mod.Oracle(full, {"t": np.arange(3.0), "a": np.ones(3), "dadt": np.ones(3)}, 1.0)


def points(values, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(-1.7, 1.7, (32 * 3 * len(values), 3))
    for k, x in enumerate(values):
        for d in range(3):
            i = 32 * (3 * k + d)
            p[i:i + 32, d] = x
    return p


def same(got, want):
    got, want = np.asarray(got, dtype=np.float32), np.asarray(want, dtype=np.float32)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    np.testing.assert_array_equal(got[ok].view(np.uint32), want[ok].view(np.uint32))


@pytest.mark.parametrize("order", [1, 2])
def test_exact_gathers(gpu_lib, pkg, full, oracle, order):
    p = points(FAR + [1e160, -1e160, 1e308], 1)
    tree = pkg.Octree.from_records(full)
    got = tree.cic(p, exact=True) if order == 1 else tree.tsc(p, exact=True)
    tree.close()
    same(got, oracle.cic(p) if order == 1 else oracle.tsc(p))
