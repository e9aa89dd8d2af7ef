"""Halo values that the sweeps only copy before they use them: any bits a caller
leaves there, those of the hand-over slots' empty mark (a signalling NaN) among
them, act as in the sequential routine."""
import numpy as np
import pytest

from conftest import gen, pkg

pytestmark = pytest.mark.gpu

MARK = np.array([0x7FF0000100000001, 0x7FF000017FF00001, 0xFFF0000100000000],
                dtype=np.uint64).view(np.float64)


def both(s, phi0, n_sweep):
    import oracle
    a, b = phi0.copy(), phi0.copy()
    with pkg().CGSolver(s.nr, s.nth, s.nz) as cg:
        cg.tdma(s.arrays(), a, n_sweep)
    with np.errstate(all="ignore"):
        oracle.tdma_3d(s, b, n_sweep)
    return a, b


@pytest.mark.parametrize("dims", [(13, 10, 9), (9, 10, 13), (40, 17, 33)])
@pytest.mark.parametrize("side", ["r", "z"])
def test_signalling_nans_beside_the_first_lines(dims, side):
    g = gen()
    s = g.make_transport_system(*dims, seed=3)
    rng = np.random.default_rng(5)
    phi0 = rng.normal(size=g.halo_shape(*dims))
    face = phi0[2:-2, 2:-2, 1] if side == "r" else phi0[1, 2:-2, 2:-2]
    for k, v in enumerate(MARK):
        face[k + 1, 2 * k + 1] = v
    a, b = both(s, phi0, 2)
    live = ~np.isnan(b)
    assert np.isnan(b).any() and live.any()
    assert np.array_equal(np.isnan(a), ~live)
    assert np.array_equal(a[live].view(np.uint64), b[live].view(np.uint64))


@pytest.mark.parametrize("dims", [(37, 20, 33), (12, 24, 16), (1, 9, 20)])
def test_signs_of_zeros(dims):
    """Right-hand sides of -0 and links that vanish: the results' zeros carry
    the sequential routine's signs."""
    g = gen()
    s = g.make_transport_system(*dims, seed=9)
    rng = np.random.default_rng(1)
    inner = lambda a: a[2:-2, 2:-2, 2:-2]  # noqa: E731
    zero = rng.random(inner(s.Su).shape) < 0.3
    inner(s.Su)[zero] = -0.0
    for n in ("aW", "aE", "aS", "aN", "aB", "aT"):
        inner(getattr(s, n))[zero] = 0.0
    phi0 = rng.normal(size=g.halo_shape(*dims))
    a, b = both(s, phi0, 2)
    assert not np.isnan(b).any() and (inner(b) == 0.0).any()
    assert np.array_equal(a.view(np.uint64), b.view(np.uint64))
