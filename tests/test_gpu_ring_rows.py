"""Line of sight z with the ring table in CTAs of 32 to 256 rows: sides at which the rows
per CTA are the least, in between, fill one wave and several, against the oracle's float64
sums over the same transforms.

Tolerance, of the bin's monopole: a mode's power has 16 ulps from three MAS factors (each an
ulp and a rounding) and two products, up to 25 in its Legendre factor; a float32 partial sum of
at most 4096 terms has 64 with independent roundings: (64 + 64) * 2^-24, times 2 l + 1 = 9."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dims,fields', [(2, 1), (31, 1), (64, 2), (129, 1), (130, 4), (200, 2), (300, 1), (448, 2)])
def test_ring_rows(dims, fields):
    import pylians_gb300.build as b
    b.build()
    import pylians_gb300.Pk_library as PKL
    r = np.random.default_rng(dims)
    d = [r.standard_normal((dims,) * 3).astype(np.float32) for _ in range(fields)]
    mas = ['TSC', 'CIC', 'NGP', 'PCS'][:fields]
    sums = O.pk_mode_sums([PKL.FFT3Dr_f(x) for x in d], 2, [O.MAS_function(m) for m in mas], 8)
    ref = O.finalize_pk(sums, 1000.0, dims, fields, cross=fields > 1)
    got = PKL.XPk(d, 1000.0, 2, mas) if fields > 1 else PKL.Pk(d[0], 1000.0, 2, mas[0])
    shape = (-1, 3, fields)
    got3, ref3 = got.Pk.reshape(shape), ref.Pk.reshape(shape)
    got2, ref2 = got.Pk2D.reshape(-1, fields), ref.Pk2D.reshape(-1, fields)
    assert np.array_equal(got.Nmodes3D, ref.Nmodes3D) and np.array_equal(got.Nmodes2D, ref.Nmodes2D)
    tol = 128 * 2.0 ** -24
    assert (np.abs(got3 - ref3) <= 9 * tol * ref3[:, :1]).all()
    some = ref.Nmodes2D > 0
    assert (np.abs(got2 - ref2) <= tol * ref2)[some].all()
