"""The block operations of the device vectors (sf_vecs_gram, sf_vecs_update)
against numpy in FP64, at the edges of their tiles: one vector, counts below,
at and past 8, 16 and 32, 2D and 3D, a height that is no multiple of a chunk of
8 levels. The padding of a level's row (modes past K1 K2) holds NaN: it takes
no part in a dot product.

Bounds: a dot product is the FP64 sum of exact products of floats times a
quadrature weight (held in 32 bits), so it agrees with numpy's to the rounding
of FP64 sums, 1e-12 of the norms; an update adds na products in FP32, in
partial sums of at most na / 8 + 8 terms, so its error is at most about
(na / 8 + 8) 2^-24 of the sum of the terms' magnitudes."""
import numpy as np
import pytest

from tests.helpers import CONFIGS
from tests.test_gpu_parity import gpu_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n2,n3", [(1, 64), (1, 44), (16, 36)])
@pytest.mark.parametrize("na,nb", [(1, 1), (3, 4), (16, 8), (17, 9), (32, 16), (33, 17), (65, 32)])
def test_gram_and_update_match_numpy(n2, n3, na, nb):
    import stratiflow_b200 as sf
    from stratiflow_b200.grid import vertical_points, vertical_points_fractional
    cfg = dict(CONFIGS["lin2d"], N2=n2, N3=n3)
    s = gpu_solver(cfg)
    P, rng = s.K1 * s.K2, np.random.default_rng(3)
    x = (rng.normal(size=(na + nb,) + (5, n3, s.plane)) + 1j * rng.normal(size=(na + nb,) + (5, n3, s.plane))).astype(np.complex64)
    if n2 == 1:
        x[:, 1] = 0
    x[..., P:] = np.nan
    v = sf.Vecs(s, na + nb)
    for i in range(na + nb):
        v.set(i, x[i])
    z, zf = vertical_points(cfg["L3"], n3), vertical_points_fractional(cfg["L3"], n3)
    wn, wd = np.zeros(n3), np.zeros(n3)
    wn[1:n3 - 1] = z[2:] - z[1:n3 - 1]
    wd[2:n3 - 1] = zf[2:n3 - 1] - zf[1:n3 - 2]
    w = np.stack([wn, wn, wd, 0.2 * wn]).astype(np.float32).astype(np.float64)
    w[3] = wn.astype(np.float32).astype(np.float64) * 0.2
    wm = np.full(P, 2.0)
    wm[0] = 1.0
    d = x[:, :4, :, :P].astype(np.complex128)
    c = np.einsum("ifzm,kfzm,fz,m->ik", d[:na], d[na:].conj(), w, wm, optimize=True).real
    norm = np.sqrt(np.einsum("ifzm,fz,m->i", np.abs(d) ** 2, w, wm))
    got = v.gram(0, na, v, na, nb, 0.2)
    assert np.max(np.abs(got - c) / (norm[:na, None] * norm[None, na:])) < 1e-12
    coef = rng.normal(size=(na, nb))
    v.update(na, nb, -0.5, v, 0, na, coef)
    ref = d[na:] - 0.5 * np.einsum("ik,ifzm->kfzm", coef, d[:na])
    mag = np.abs(d[na:]) + 0.5 * np.einsum("ik,ifzm->kfzm", np.abs(coef), np.abs(d[:na]))
    for k in range(nb):
        out = v.get(na + k)[:4, :, :P]
        assert np.max(np.abs(out - ref[k]) / mag[k].clip(1e-30)) < 2 * (na / 8 + 8) * 2.0 ** -24
    del v
    s.close()
