"""The native finalisation of P(k) sums against numpy float64 expressions of
Pk_library.pyx:384-421 and :740-796: the same bits, for one to four fields, odd and even
sides, empty bins and BoxSize as float, int and float32."""
import numpy as np
import pytest

import pylians_gb300.build as b


def _numpy(s, g, box, dims, F, cross):
    import pylians_gb300.Pk_library as PKL
    kF, kN, np1, nq, n3 = PKL.frequencies(box, dims)
    s, g = PKL._split_sums(s, dims, F), PKL._split_geometry(g, dims)
    fact = (box / dims ** 2) ** 3
    N1, N2, N3 = g['N1'][1:], g['N2'], g['N3'][1:]
    with np.errstate(all='ignore'):
        k1D = (g['K1'][1:] / N1) * kF
        area = (np.pi * np.sqrt(kN ** 2 - k1D ** 2) ** 2 / N1) / (2.0 * np.pi) ** 2
        P1 = s['P1'][1:] * fact * area[:, None]
        P2 = s['P2'] * fact / N2[:, None]
        P3 = (s['P3'][1:] * np.array([1.0, 5.0, 9.0])[:, None] / N3[:, None, None]) * fact
        r = dict(k1D=k1D, Nmodes1D=N1, Nmodes2D=N2, Nmodes3D=N3, k3D=(g['K3'][1:] / N3) * kF,
                 kpar=np.tile(0.5 * (2 * np.arange(np1 + 1) + 1) * kF, nq + 1),
                 kper=np.repeat(0.5 * (2 * np.arange(nq + 1) + 1) * kF, np1 + 1))
        if cross:
            r.update(Pk1D=P1[:, :F], PkX1D=P1[:, F:], Pk2D=P2[:, :F], PkX2D=P2[:, F:], Pk=P3[..., :F], XPk=P3[..., F:])
        else:
            r.update(Pk1D=P1[:, 0], Pk2D=P2[:, 0], Pk=P3[..., 0], Pkphase=(s['PH'][1:, 0] / N3) * fact)
    return r


@pytest.mark.parametrize('F,cross', [(1, False), (1, True), (2, True), (4, True)])
@pytest.mark.parametrize('dims,box', [(1, 1.0), (2, 75.3), (3, 1000), (16, 0.1), (65, np.float32(333.3)), (128, 1e3)])
def test_finalize_bits(dims, box, F, cross):
    b.build()
    import pylians_gb300.Pk_library as PKL
    _, _, p, q, k = PKL.frequencies(1.0, dims)
    nb1, nb2, nb3, C = p + 1, (p + 1) * (q + 1), k + 1, F + F * (F - 1) // 2
    r = np.random.default_rng(dims)
    s = r.lognormal(size=(3 * nb3 + nb1 + nb2) * C + nb3 * F)
    g = r.integers(0, 9, 2 * nb1 + nb2 + 2 * nb3).astype(np.float64)
    g[:nb1] *= 0.77
    own = 1 if dims % 2 else 8
    g[-nb3] += (dims ** 3 - own) // 2 + own - g[-nb3:].sum()
    got, ref = PKL.finalize_pk(s, g, box, dims, F, cross).__dict__, _numpy(s, g, box, dims, F, cross)
    assert set(got) == set(ref)
    for name in ref:
        assert got[name].shape == ref[name].shape and got[name].dtype == np.float64
        assert np.array_equal(got[name], ref[name], equal_nan=True), name
    with pytest.raises(ValueError):
        PKL.finalize_pk(s[:-1], g, box, dims, F, cross)
