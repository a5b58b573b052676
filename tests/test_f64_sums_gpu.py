"""The FP64 wave update forms a pair's two sums as integer arithmetic where
the operands' exponents allow it and on the FP64 unit otherwise.  Bar: bit for
bit the oracle's fused flavour on fields whose neighbours are alike, spread over
many binades (both paths in every warp), cancel exactly or nearly, sit at the
ends of the exponent range, or are zeros, subnormals, infinities and NaN."""
import numpy as np
import pytest

import stencil3d_gb300 as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRID = (7, 19, 70, 4, 4, 4)


def _fields(kind, rng):
    shape = O.shape(GRID)
    sign = rng.choice([-1.0, 1.0], shape)
    if kind == "alike":
        u = 1.0 + 2.0 ** -30 * rng.integers(-8, 9, shape) + 2.0 ** -52 * rng.integers(0, 4, shape)
    elif kind == "random":
        u = rng.uniform(-1e-3, 1e-3, shape)
    elif kind == "spread":
        u = sign * rng.uniform(1.0, 2.0, shape) * 2.0 ** rng.integers(-12, 3, shape)
    elif kind == "cancel":
        u = sign * (1.0 + 2.0 ** -52 * rng.integers(0, 3, shape))
    elif kind == "small":
        u = sign * rng.uniform(1.0, 2.0, shape) * 2.0 ** rng.integers(-1030, -955, shape).astype(float)
    elif kind == "large":
        u = sign * rng.uniform(1.0, 2.0, shape) * 2.0 ** rng.integers(1012, 1020, shape).astype(float)
    else:
        u = rng.uniform(-1.0, 1.0, shape)
        at = rng.integers(0, 40, shape)
        for n, x in enumerate((0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2e-308)):
            u[at == n] = x
    v = u * rng.choice([1.0, 0.75, -1.0], shape)
    return v, np.full(shape, 0.25), u


@pytest.mark.parametrize("points", [7, 13, 25])
@pytest.mark.parametrize("kind", ["alike", "random", "spread", "cancel", "small", "large", "special"])
def test_f64_wave_is_the_oracle_bit_for_bit(kind, points):
    v, s, u = _fields(kind, np.random.default_rng(points))
    src = (3, 9, 40)
    with np.errstate(all="ignore"), S.Stencil(S.Grid(*GRID), points, "wave", "f64", dt=5e-4, src=src) as st:
        vv, uu = v.copy(), u.copy()
        st.iterate_host(vv, s, uu, 3)
    c0, c1, c2 = O.wave_constants(points, 1500.0, 5e-4, 10.0)
    O.iterate_wave(u, v, s, GRID, points, 3, c0, c1, c2, src=src,
                   amps=O.ricker_amps(0, 3, 5e-4, dtype=np.float64), fma=True)
    np.testing.assert_array_equal(O.interior(uu, GRID), O.interior(u, GRID))
    np.testing.assert_array_equal(O.interior(vv, GRID), O.interior(v, GRID))
