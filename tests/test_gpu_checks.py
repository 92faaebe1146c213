"""Energy, observables and norm reductions over every row layout (rows shorter
and longer than a CTA, lengths that are no power of two, one plane and many)
against numpy in double precision.

The reductions add at most 2^20 terms of one sign (or of the size of their
absolute sum) in FP64, compensated: 1e-12 of the sum of magnitudes bounds the
order of summation and the transform's rounding (1e-14)."""
import numpy as np
import pytest

import gpue_b200 as G

pytestmark = pytest.mark.gpu


def state(dim, n, box, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = -box + box / (n >> 1) * np.arange(n)
    r2 = sum((x.reshape([-1 if k == a else 1 for k in range(dim)])) ** 2 for a in range(dim))
    psi = np.exp(-r2 / 8) * (1 + 0.1 * rng.standard_normal((n,) * dim)) * np.exp(
        1j * rng.uniform(0, 1, (n,) * dim))
    return x, psi / np.sqrt(np.sum(np.abs(psi) ** 2) * (box / (n >> 1)) ** dim)


def terms(dim, n, box, x, psi, g, omega):
    """(kinetic, potential, interaction, rotation) and the dict of moments."""
    dx = box / (n >> 1)
    dV = dx ** dim
    ax = [x.reshape([-1 if dim - 1 - k == a else 1 for k in range(dim)]) for a in range(dim)]
    V = sum(0.5 * c ** 2 for c in ax)
    if omega:
        V = V + 0.5 * ((omega * ax[1]) ** 2 + (omega * ax[0]) ** 2)
    d = np.abs(psi) ** 2
    p = np.fft.fftfreq(n, d=1.0 / n) * np.pi / box
    K = sum(0.5 * p.reshape([-1 if dim - 1 - k == a else 1 for k in range(dim)]) ** 2
            for a in range(dim))
    kin = np.sum(K * np.abs(np.fft.fftn(psi)) ** 2) / psi.size * dV

    def diff(a):
        f = psi.ravel()
        out = f / dx
        s = n ** a
        out[:-s] = (f[s:] - f[:-s]) / dx
        return out.reshape(psi.shape)

    rot = 0.0
    if omega:
        rot = np.sum((psi.conj() * 1j * (-omega * ax[1] * diff(0) + omega * ax[0] * diff(1))).real
                     ) * dV
    w = np.ones(n)
    w[0] = w[-1] = 0.5
    wd = d.copy()
    for a in range(dim):
        wd = wd * w.reshape([-1 if dim - 1 - k == a else 1 for k in range(dim)])
    lz = np.sum((psi.conj() * -1j * (ax[0] * diff(1) - ax[1] * diff(0))).real) * dV
    m = {"norm": np.sum(d) * dV, "x": np.sum(wd * ax[0]) * dV, "y": np.sum(wd * ax[1]) * dV,
         "r2": np.sum(wd * (ax[0] ** 2 + ax[1] ** 2)) * dV,
         "q": np.sum(wd * (ax[0] ** 2 - ax[1] ** 2)) * dV, "lz": lz}
    return (kin, np.sum(V * d) * dV, np.sum(0.5 * g * d * d) * dV, rot), m


@pytest.mark.parametrize("dim,n", [(2, 16), (2, 96), (2, 160), (2, 320), (2, 640), (2, 1024),
                                   (3, 16), (3, 32), (3, 96)])
@pytest.mark.parametrize("omega", [0.0, 0.6])
def test_energy_observables_and_norm(dim, n, omega):
    box, g = 6.0, 40.0
    x, psi = state(dim, n, box, 7 + n)
    p = G.make_params(dim, n, box, g=g, omega=omega, gauge=omega != 0.0)
    with G.Solver(p) as s:
        s.set_wfc(psi)
        e, o, nrm = s.energy(), s.observables(), s.norm()
    t, m = terms(dim, n, box, x, psi, g, omega)
    scale = sum(abs(v) for v in t) + 50 * abs(m["norm"])
    assert abs(e - sum(t)) < 1e-12 * scale
    for key, v in zip(("e_kinetic", "e_potential", "e_interaction", "e_rotation"), t):
        assert abs(o[key] - v) < 1e-12 * scale, key
    for key, v in m.items():
        assert abs(o[key] - v) < 1e-12 * scale, key
    assert abs(nrm - m["norm"]) < 1e-12 * m["norm"]


@pytest.mark.parametrize("prec,tol", [(G.PREC_FP64, 1e-12), (G.PREC_FP32, 1e-6)])
@pytest.mark.parametrize("dim,n", [(2, 16), (2, 192), (2, 1024), (3, 32), (3, 128)])
def test_norm_that_evolve_returns(dim, n, prec, tol):
    """The norm that comes with the final renormalisation is that of the state
    returned, which is normalised."""
    _, psi = state(dim, n, 6.0, 3)
    with G.Solver(G.make_params(dim, n, 6.0, g=40.0, gdt=1e-4, precision=prec)) as s:
        s.set_wfc(psi)
        r = s.evolve(3, 0)
        out = s.get_wfc()
        nrm = s.norm()
    dV = (6.0 / (n >> 1)) ** dim
    assert abs(r["norm"] - np.sum(np.abs(out) ** 2) * dV) < 1e-12
    assert abs(r["norm"] - nrm) < 1e-14 and abs(nrm - 1) < tol
