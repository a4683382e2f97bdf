"""The spinful row generator's short route (even nphi: the untranslated row state stands for its translates) against
the general formula, which sums over every translate of the row state (BLQH_with_spin/lanczos_hamiltonian.cpp:86-927).

The general formula is restated here in Python; its short form is compared with it on the CPU, and the GPU's rows
with it for every kind of term: tunnelling, twists, parallel field, odd electron numbers, odd nphi, no symmetry.
Values: at most ~60 terms of size <= 2 per entry, each to 2^-52: 2e-14."""
import itertools
import math

import numpy as np
import pytest

from oracle.spin_ref import translate

# (nphi, nel, nel_up, nel_su, J, K), (d, dsas, dv, dz, theta_b, theta_x, theta_y)
CASES = [
    ((4, 4, 2, 2, 0, 0), (0.7, 0.0, 0.01, 0.02, 0.0, 0.0, 0.0)),
    ((4, 4, 2, 2, 2, 2), (0.7, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)),
    ((4, 4, 2, 2, 1, 1), (1.3, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)),
    ((4, 4, -1, -1, 0, 1), (1.1, 0.2, 0.01, 0.02, 0.0, 0.0, 0.0)),
    ((4, 4, -1, 2, 2, 2), (1.1, 0.2, 0.0, 0.0, 0.0, 0.0, 0.0)),
    ((4, 3, 1, 1, 2, 3), (0.5, 0.0, 0.0, 0.1, 0.0, 0.0, 0.0)),
    ((4, 4, -1, -1, 0, 0), (0.9, 0.3, 0.0, 0.0, 0.4, 0.0, 0.0)),  # parallel field with tunnelling
    ((4, 4, 2, 2, 0, 1), (0.9, 0.0, 0.0, 0.0, 0.4, 0.0, 0.0)),    # parallel field alone
    ((4, 4, 2, 2, 0, 2), (0.9, 0.0, 0.0, 0.0, 0.0, 0.3, 0.0)),    # twist theta_x
    ((4, 4, 2, 2, 0, 1), (0.9, 0.0, 0.0, 0.0, 0.0, 0.0, 0.5)),    # twist theta_y
    ((6, 3, 1, 2, 0, 3), (0.8, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)),
    ((3, 3, -1, -1, 0, 1), (0.8, 0.1, 0.0, 0.0, 0.0, 0.0, 0.0)),  # odd nphi
    ((5, 3, 1, 1, 2, 0), (0.8, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)),
    ((4, 3, 1, 1, 2, -1), (0.8, 0.0, 0.01, 0.0, 0.0, 0.0, 0.0)),  # no translation symmetry
]


def tables(nphi, d, theta_x):
    """V[inter][s][|t|] and the background energy (BLQH_with_spin/lanczos_hamiltonian.cpp:45-85)."""
    l = math.sqrt(2 * math.pi * nphi)
    V = np.zeros((2, nphi, nphi))
    s = np.arange(nphi)
    top = 10 * nphi / (d + 0.01)
    for a, xs in ((0, range(-nphi, nphi + 1)), (1, range(int(-top), math.ceil(top)))):
        for qy in range(nphi):
            for qx in xs:
                if qx == 0 and qy == 0:
                    continue
                q = 2 * math.pi * math.sqrt(qx * qx + qy * qy) / l
                f = 2 * math.pi / q * math.exp(-q * q / 2 - (q * d if a else 0.0))
                V[a, :, qy] += 2 * f * np.cos((2 * np.pi * s - (theta_x if a else 0.0)) * qx / nphi) / (2 * l * l)
    ec = -2.0 + sum(math.erfc(math.sqrt(math.pi * (i * i + j * j))) for i in range(nphi) for j in range(nphi) if i or j)
    return V, ec / l


def empties(c, a, b):
    return sum(1 for o in range(a + 1, b) if not (c >> o) & 1)


def moves(c, nphi, par, V):
    """(target, amplitude) of every move from state c, signs included."""
    d, dsas, _, _, theta_b, _, theta_y = par
    occ = [o for o in range(4 * nphi) if (c >> o) & 1]
    for n, m in itertools.combinations(occ, 2):
        ba, bb = n // nphi, m // nphi
        inter = (ba // 2) != (bb // 2)
        rest = c & ~(1 << n) & ~(1 << m)
        for t in range(-(nphi - 1), nphi):
            nt, mt = ba * nphi + (n % nphi + t) % nphi, bb * nphi + (m % nphi - t) % nphi
            if nt == mt or (rest >> nt) & 1 or (rest >> mt) & 1:
                continue
            sg = empties(rest, min(n, nt), max(n, nt)) + empties(rest, min(m, mt), max(m, mt)) + (nt > mt)
            v = V[int(inter), abs(mt % nphi - n % nphi), abs(t)] * (-1) ** sg
            if inter and ba % 2 != bb % 2:
                v = v * complex(math.cos(theta_y * t / nphi), math.sin(theta_y * t / nphi))
            yield rest | (1 << nt) | (1 << mt), v
    if dsas > 0:
        for r in range(nphi):
            for n, nt, amp, ph in ((r, r + 2 * nphi, 0.25, theta_b * r * d), (2 * nphi + r, r, 0.25, -theta_b * r * d),
                                   (nphi + r, 3 * nphi + r, 0.25, theta_b * r * d),
                                   (3 * nphi + r, nphi + r, 0.25, -theta_b * r * d),
                                   (r, 3 * nphi + r, 0.5, 0.0), (nphi + r, 2 * nphi + r, 0.5, 0.0)):
                if ((c >> n) & 1) != ((c >> nt) & 1):
                    sg = empties(c, min(n, nt), max(n, nt))
                    yield c ^ (1 << n) ^ (1 << nt), -amp * dsas * (-1) ** sg * complex(math.cos(ph), math.sin(ph))


def basis(sec):
    """Smallest members of the orbits that momentum J meets, their periods."""
    nphi, nel, up, su, J, K = sec
    out = []
    for occ in itertools.combinations(range(4 * nphi), nel):
        c = sum(1 << o for o in occ)
        nb = [bin((c >> (b * nphi)) & ((1 << nphi) - 1)).count("1") for b in range(4)]
        if (J >= 0 and sum(o % nphi for o in occ) % nphi != J) or (up >= 0 and nb[0] + nb[1] != up):
            continue
        orbit = [translate(c, k, nphi)[0] for k in range(nphi)] if K >= 0 else [c]
        mom = [sum(o % nphi for o in range(4 * nphi) if (x >> o) & 1) % nphi for x in orbit]
        if c != min(x for x, q in zip(orbit, mom) if J < 0 or q == J) or (su >= 0 and nb[0] + nb[2] != su):
            continue
        period = next((k for k in range(1, nphi) if orbit[k] == c), nphi) if K >= 0 else nphi
        out.append((c, period))
    return sorted(out)


def matrix(states, sec, par, short):
    """The reference's row sums; short: untranslated moves, each with the sum over the row's translates."""
    nphi, nel, _, _, _, K = sec
    d, _, dv, dz = par[:4]
    V, ec = tables(nphi, d, par[5])
    where = {}
    for j, (c, P) in enumerate(states):
        for k in range(P if K >= 0 else 1):
            where[translate(c, k, nphi)[0]] = (j, k)
    H = np.zeros((len(states), len(states)), complex)

    def ft(m):
        return complex(math.cos(2 * math.pi * m * K / nphi), math.sin(2 * math.pi * m * K / nphi)) if K > 0 else 1.0

    for i, (c, P) in enumerate(states):
        Dl = P if K >= 0 else 1
        for ql in range(1 if short else Dl):
            lb, pl = translate(c, ql, nphi)
            for x, v in moves(lb, nphi, par, V):
                if x not in where:
                    continue
                j, k = where[x]
                Dr = states[j][1] if K >= 0 else 1
                if short:
                    g = 0.0
                    for q in range(Dl):
                        y, p1 = translate(x, q, nphi)
                        k2 = (k + q) % Dr
                        g += p1 * translate(y, k2, nphi, inverse=True)[1] * ft(q - k2)
                else:
                    g = pl * translate(x, k, nphi, inverse=True)[1] * ft(ql - k)
                H[i, j] += v * g / math.sqrt(Dl * Dr)
        n = [bin((c >> (b * nphi)) & ((1 << nphi) - 1)).count("1") for b in range(4)]
        H[i, i] += ec * nel - d * (n[0] + n[1]) * (n[2] + n[3]) / nphi - 0.5 * dv * (n[0] + n[1] - n[2] - n[3]) \
            - 0.5 * dz * (n[0] + n[2] - n[1] - n[3])
    H[np.abs(H) <= 1e-10] = 0
    return H


def covariant(sec, par):
    return sec[5] < 0 or (sec[0] % 2 == 0 and par[5] == 0.0 and not (par[4] != 0.0 and par[1] > 0))


@pytest.mark.parametrize("sec,par", CASES, ids=str)
def test_short_form_equals_sum_over_translates(sec, par):
    """On the CPU, where the route is taken."""
    states = basis(sec)
    assert states
    if covariant(sec, par):
        a, b = matrix(states, sec, par, False), matrix(states, sec, par, True)
        assert np.max(np.abs(a - b)) < 2e-14


@pytest.mark.gpu
@pytest.mark.parametrize("sec,par", CASES, ids=str)
def test_rows_on_gpu(sec, par):
    import blqh_gb300 as B

    states = basis(sec)
    b = B.basis_spin(*sec, rep_mode=B.REP_MIN)
    assert [int(x) for x in b.id] == [c for c, _ in states]
    d, dsas, dv, dz, tb, tx, ty = par
    H = B.hamiltonian_spin(b, d, dsas, dv, dz, theta_b=tb, theta_x=tx, theta_y=ty)
    rp, col, val = H.csr()
    D = np.zeros((H.dim, H.dim), complex)
    D[np.repeat(np.arange(H.dim), np.diff(rp)), col] = val
    ref = matrix(states, sec, par, False)
    if not H.is_complex:
        ref = ref.real
    assert np.array_equal(D != 0, ref != 0)
    assert np.max(np.abs(D - ref)) < 2e-14
