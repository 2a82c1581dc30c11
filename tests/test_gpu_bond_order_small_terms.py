"""Bond-order forces that are small: an atom at 3 to 7 angstrom from a bonded pair,
where the cutoff function is 1e-3 to 1e-10, against the formulas in extended
precision, relative to each atom's own force.  (The oracle and the reference form
the cutoff as (1 - tanh) / 2, which is off by 5e-17 of 1 whatever its size: not
exact enough here.)  Bar: distances rounded to 2^-53 change the cutoff's exponent
by 4 x 7 units (3e-15), the far angle's cosine multiplies roundings by the ratio
of the sides (6), and a dozen such terms add: 1e-13 at most, a tenth of it usual."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _f(x):
    return LD(float(np.float32(x)))


def _cut(r):
    fc = 1 / (1 + np.exp(4 * (r - _f(1.3))))
    return fc, -4 * fc * (1 - fc)


def _angle(c):
    q = _f(4.0417) + c * c
    k = LD(float(np.float32(1) + np.float32(25) / np.float32(4.0417)))
    return k - 25 / q, 50 * c / (q * q)


def _forces(pos):
    """Forces on three atoms that are all candidates of one another."""
    x, t = pos[:, :3].astype(LD), pos[:, 3].astype(int)
    F = np.zeros((3, 3), LD)
    for i, j, m in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)):
        dij, dim, djm = x[i] - x[j], x[i] - x[m], x[j] - x[m]
        rij, rim, rjm = (np.sqrt((d * d).sum()) for d in (dij, dim, djm))
        same = t[i] == t[j]
        re, de, be, r0 = ((1.097, 941.4e-4, 2.71009, 3.72) if same and t[i] == 0 else
                          (1.2075, 493.55309e-4, 2.2478, 3.31) if same else
                          (1.15, 626.734e-4, 2.24068, 3.51))
        re, de, be, r0 = _f(re), _f(de), _f(be), _f(r0)
        va = 2 * de * np.exp(-be * (rij - re))
        vr2 = de * np.exp(-2 * be * (rij - re)) + _f(7.0e-8) * np.exp(-10 * be * (rij - re))
        gm = np.float32(0.3)
        ep, gx = np.exp(3 * (rij - r0)), LD(float(gm)) * np.exp(-3 * (rij - r0))
        A, B = ep + gx, 3 * (ep - gx)
        k10 = LD(float(np.float32(10) * (gm - np.float32(1))))
        v = LD(float(np.float32(1) + np.float32(50) * gm + np.float32(0.09))) + k10 * B
        dvdw = -_f(1.0e-4) * ((k10 * 9 * A * A - 2 * B * v) / (A * A * A))
        lam, E = _f(1.33), np.exp(_f(1.33) * (rij - re))
        (fi, dfi), (fj, dfj) = _cut(rim), _cut(rjm)
        ci = (dij * dim).sum() / (rij * rim)
        cj = -(dij * djm).sum() / (rij * rjm)
        (gi, pi), (gj, pj) = _angle(ci), _angle(cj)
        bi, bj = 1 / (1 + fi * gi * E), 1 / (1 + fj * gj * E)
        # derivatives of xi_ij and xi_ji along u_im and u_ij (r_i moved)
        ai = E * (dfi * gi + fi * pi * (1 / rij - ci / rim))
        aj = -E * fj * pj * rim / (rij * rjm)
        ui = E * fi * (pi * (1 / rim - ci / rij) + gi * lam)
        uj = E * fj * (pj * (1 / rjm - cj / rij) + gj * lam)
        uij, uim = dij / rij, dim / rim
        db = (bi * bi * (ai * uim + ui * uij) + bj * bj * (aj * uim + uj * uij)) / 2
        F[i] += (2 * be * vr2 - (bi + bj) / 2 * be * va + dvdw) * uij - va * db
        # and the force on the third body
        wi, wj = va * E * bi * bi / 4, va * E * bj * bj / 4
        F[m] += (wi * ai / E + wj * aj / E) * uim
        F[m] += djm / rjm * (-wi * fi * pi * rjm / (rij * rim) +
                             wj * (dfj * gj + fj * pj * (1 / rij - cj / rjm)))
    return F


@pytest.mark.parametrize("d", [3.0, 4.0, 5.0, 6.0, 7.0])
@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_force_on_a_far_atom(eng, d, seed):
    rng = np.random.default_rng(seed)
    u = rng.standard_normal((2, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    pos = np.zeros((3, 4))
    pos[1, :3] = 1.2 * u[0]
    pos[2, :3] = d * u[1]
    pos[:, :3] -= pos[:, :3].mean(0)
    pos[1, 3] = seed % 2
    cfg = eng.make_config(n_mb=3, use_lj=0, use_mb=1, mb_rs=9.9, mb_rcut=9.8, dt=0.5, species=0)
    with eng.Engine(cfg) as e:
        e.upload(pos, np.zeros((3, 3)))
        e.begin(0.0)
        p, _ = e.download()
        f, _ = e.compute_forces()
    ref = _forces(p)
    err = np.linalg.norm((f - ref).astype(float), axis=1) / np.linalg.norm(ref.astype(float), axis=1)
    assert err.max() < 1e-13, err
