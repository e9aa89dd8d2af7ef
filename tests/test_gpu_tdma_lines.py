"""Line lengths, owner counts and operators at the edges of the device TDMA's
segmented line solve: a warp's lanes own ceil(L/32) elements each (sizes around
multiples of 32 and at the instantiated maxima), blocks own several adjacent
lines' chains, and a grid may walk its owners in rounds. The sweeps stay the
sequential routine's, so every comparison is bit for bit over the whole array."""
import numpy as np
import pytest

from conftest import gen, pkg

pytestmark = pytest.mark.gpu


def both(s, phi0, n_sweep):
    import oracle
    a, b = phi0.copy(), phi0.copy()
    with pkg().CGSolver(s.nr, s.nth, s.nz) as cg:
        cg.tdma(s.arrays(), a, n_sweep)
    with np.errstate(all="ignore"):
        oracle.tdma_3d(s, b, n_sweep)
    return a, b


def rand_phi(dims, seed):
    return np.random.default_rng(seed).normal(size=gen().halo_shape(*dims))


@pytest.mark.parametrize("dims", [(31, 32, 33), (64, 65, 9), (9, 96, 97), (128, 7, 129),
                                  (10, 160, 161), (193, 224, 5), (5, 256, 257), (3, 385, 6),
                                  (513, 4, 3), (2, 3, 769), (2, 1024, 3), (40, 1, 17),
                                  (17, 2, 40)])
def test_line_lengths(dims):
    s = gen().make_transport_system(*dims, seed=3)
    a, b = both(s, rand_phi(dims, 5), 2)
    assert np.array_equal(a, b)


def test_more_owners_than_blocks():
    """Long r lines leave one owner a block: 200 owners walk 148 SMs in rounds."""
    dims = (1000, 2, 200)
    s = gen().make_transport_system(*dims, seed=11)
    a, b = both(s, rand_phi(dims, 1), 2)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("dims", [(35, 70, 50), (60, 40, 96)])
def test_weakly_contracting_lines(dims):
    """Lines whose recurrences forget their start slowly (links of a line
    direction 1e6 times the others, no sink): many passes per line."""
    s = gen().make_transport_system(*dims, seed=7, trivial_frac=0.0, peclet=0.0, sp_frac=0.0)
    for n in ("aW", "aE"):
        getattr(s, n)[...] *= 1e6
    links = sum(getattr(s, n) for n in ("aW", "aE", "aS", "aN", "aB", "aT"))
    s.aP[...] = np.where(s.aP != 0.0, links, s.aP)
    a, b = both(s, rand_phi(dims, 2), 2)
    assert np.array_equal(a, b)


def test_pressure_operator_lines():
    """Density contrast 26,000:1: links of a line over ten decades."""
    s = gen().make_system(35, 70, 50, 16, seed=4)
    a, b = both(s, rand_phi((35, 70, 50), 3), 2)
    assert np.array_equal(a, b)


def test_extreme_operands():
    """Pivots and sources outside the reciprocal's range, exact zeros of both
    signs, overflow to infinity and NaN: the same values and the same
    non-finite cells."""
    dims = (37, 20, 33)
    s = gen().make_transport_system(*dims, seed=9)
    rng = np.random.default_rng(1)
    inner = lambda a: a[2:-2, 2:-2, 2:-2]  # noqa: E731
    for scale in (1e-200, 1e200):
        hit = rng.random(inner(s.aP).shape) < 0.01
        inner(s.aP)[hit] *= scale
        inner(s.Su)[rng.random(hit.shape) < 0.01] *= scale
    inner(s.Su)[rng.random(inner(s.Su).shape) < 0.05] = -0.0
    phi0 = rand_phi(dims, 4)
    a, b = both(s, phi0, 1)
    assert np.array_equal(a, b, equal_nan=True)
    assert np.array_equal(np.signbit(a), np.signbit(b)) or np.isnan(b).any()
    inner(s.Su)[5, 5, 36] = np.inf
    inner(s.Su)[20, 9, 7] = np.nan
    a, b = both(s, phi0, 1)
    assert np.isnan(b).any()
    assert np.array_equal(a, b, equal_nan=True)
