"""Timed cases of the exact-diagonalization library: the calls a user's program makes.

Every case goes through blqh_gb300's public entry points and returns what they
return: energies, ground states, bases, observables, gradients. Parameters that
a user varies (layer distance, aspect ratio, start vector, training targets)
come from the seed.

Kinds:
  ground  ground_state(): sector basis -> CSR -> Lanczos -> Ritz vector -> energy
          of a spinless bilayer sector, the whole path of one parameter point
  spin    the spinful bilayer: basis, Hamiltonian, Lanczos, ground state,
          energy and observables, stage by stage
  mono    ground_state_mono(): one monolayer sector
  batch   Batch: every K-sector of one momentum at several parameter points in
          one persistent launch
  mlp     the learned start vector: loss and gradient over the training points
          (forward and backward), and a prediction (forward)
"""
import math

import numpy as np
import torch

import blqh_gb300 as B

# ---------------------------------------------------------------------------
# cases


def _ground(nphi, nel, nel_up, J, K, precision="f64", steps=200, tol=0.0, delta_sas=0.0, delta_v=0.0, start=False):
    return dict(kind="ground", nphi=nphi, nel=nel, nel_up=nel_up, J=J, K=K, precision=precision, steps=steps, tol=tol,
                delta_sas=delta_sas, delta_v=delta_v, start=start)


def _spin(nphi, nel, nel_up, nel_su, J, K, steps=200, tol=0.0):
    return dict(kind="spin", nphi=nphi, nel=nel, nel_up=nel_up, nel_su=nel_su, J=J, K=K, steps=steps, tol=tol)


def _mono(nphi, nel, J, K, steps=200, tol=0.0):
    return dict(kind="mono", nphi=nphi, nel=nel, J=J, K=K, steps=steps, tol=tol)


def _batch(nphi, nel, nel_up, J, sectors, points, precision="f32", steps=150):
    return dict(kind="batch", nphi=nphi, nel=nel, nel_up=nel_up, J=J, sectors=sectors, points=points,
                precision=precision, steps=steps)


def _mlp(nphi, nel, nel_up, points, width=256):
    return dict(kind="mlp", nphi=nphi, nel=nel, nel_up=nel_up, points=points, width=width)


def listed():
    """Sizes from the README sector (Nphi = 8), the headline configuration (Nphi = 16, 8 + 8), the Nphi = 14
    sweep, the batched sweep at Nphi = 12, the Nphi = 30 monolayer and the spinful fixtures. A fixed number of
    Lanczos steps (tol = 0, as the reference's lambda; 200 is its default) gives ground states converged to
    rounding; calls with a tolerance stop at the energy's convergence and return no ground state."""
    cases = {
        # the README sector (79 states): the smallest call, bounded by launches and latency
        "n8_readme_f64": _ground(8, 8, 4, 4, 4, tol=1e-12),
        # free layer split with tunnelling and bias, odd electron number, complex sector (1,430 states)
        "n8_free_tunnel_f64": _ground(8, 7, -1, 3, 1, tol=1e-12, delta_sas=0.1, delta_v=0.01),
        # a mid-size point of a parameter scan (5,940 states)
        "n12_f64": _ground(12, 12, 6, 0, 0),
        # one point of the all-sector Nphi = 14 sweep: complex FP64 (60k states)
        "n14_complex_f64": _ground(14, 14, 7, 0, 3),
        # the headline sector: FP32 values, FP64 vectors (647k states, 2.4e8 nonzeros)
        "n16_mixed": _ground(16, 16, 8, 0, 0, "f32", start=True),
        # a complex sector of the headline configuration (224 of its 256 sectors are complex): the largest call
        "n16_complex_mixed": _ground(16, 16, 8, 0, 1, "f32", start=True),
        # the same headline sector with FP64 values, the plain method
        "n16_f64": _ground(16, 16, 8, 0, 0, start=True),
        # spinful bilayer of the batched configuration (474 states)
        "spin6": _spin(6, 6, 3, 3, 0, 0, steps=100),
        # the largest spinful sector of the fixtures, complex (16k states)
        "spin8_complex": _spin(8, 8, 4, 4, 1, 3),
        # the Laughlin filling 1/3 at Nphi = 30, complex (100k states)
        "mono30_complex": _mono(30, 10, 0, 3),
        # a sweep: the 12 K-sectors of one J at 8 parameter points (96 instances of 5.9k states)
        "batch12_mixed": _batch(12, 12, 6, 0, 12, 8),
        # training of the learned start: 13 parameter points of the Nphi = 14 sector (780k rows)
        "mlp14": _mlp(14, 14, 7, 13),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def draw(rng):
    kind = rng.choice(["ground"] * 6 + ["spin", "mono", "mono", "batch", "mlp"])
    if kind == "ground":
        while True:
            if rng.random() < 0.12:  # odd Nphi: every translate of a row is enumerated
                nphi = rng.choice([7, 9, 11])
                nel = rng.randint(4, 6)
                up = nel // 2
            else:
                nphi = rng.choice([8, 10, 12, 14, 16])
                nel = rng.randint(max(4, nphi // 2), nphi)
                up = nel // 2 if rng.random() < 0.6 else max(1, nel // 2 - rng.randint(1, 2))
            free = nphi <= 10 and nel <= 8 and nphi % 2 == 0 and rng.random() < 0.25
            sym = not (nphi <= 10 and rng.random() < 0.1)  # now and then without translation symmetry
            J = rng.randrange(nphi)
            K = rng.choice([0, nphi // 2, rng.randrange(nphi), rng.randrange(nphi)]) if sym else -1
            prec = "f32" if rng.random() < 0.5 else "f64"
            c = _ground(nphi, nel, -1 if free else up, J, K, prec, start=rng.random() < 0.3)
            c["delta_sas"] = round(rng.uniform(0.01, 0.2), 3) if free else 0.0
            c["delta_v"] = round(rng.uniform(0.0, 0.05), 3) if rng.random() < 0.3 else 0.0
            dim, row = _size(c)
            cost = dim * row * (4 if _complex(c) else 1) * (2 if prec == "f64" else 1)
            if 40 <= dim and cost < 2.5e8:  # at most the headline sector in FP32
                if dim < 3000:
                    c["tol"] = 1e-12  # 200 steps would exhaust the Krylov space of a small sector
                return c
    if kind == "spin":
        while True:
            nphi = rng.choice([4, 6, 8])
            nel = rng.randint(3, 8)
            up = nel // 2
            su = rng.randint(max(0, nel // 2 - 1), nel // 2)
            c = _spin(nphi, nel, up, su, rng.randrange(nphi), rng.randrange(nphi))
            dim, row = _size(c)
            if 120 <= dim <= 17000:
                c["steps"] = 60 if dim < 300 else 100 if dim < 3000 else 200
                return c
    if kind == "mono":
        while True:
            nphi = rng.randint(12, 30)
            nel = rng.randint(4, 10)
            C = math.gcd(nel, nphi)
            c = _mono(nphi, nel, rng.randrange(nphi), rng.randrange(C))
            dim, row = _size(c)
            if 120 <= dim <= 110000 and math.comb(nphi, nel) <= 31e6:
                c["steps"] = 60 if dim < 300 else 100 if dim < 3000 else 200
                return c
    if kind == "batch":
        nphi = rng.choice([8, 10, 12])
        nel = rng.choice([nphi - 2, nphi])
        return _batch(nphi, nel, nel // 2, rng.randrange(nphi), rng.randint(2, nphi), rng.randint(2, 8),
                      "f64" if nphi < 12 and rng.random() < 0.4 else "f32", 150 if nphi == 12 else 60)
    nphi = rng.choice([8, 10, 12, 14])
    return _mlp(nphi, nphi, nphi // 2 - rng.randint(0, 2), rng.randint(2, 13), rng.choice([64, 128, 256]))


# ---------------------------------------------------------------------------
# sizes


def _complex(c):
    if c["kind"] == "mono":
        n = math.gcd(c["nel"], c["nphi"])
        return not (c["K"] <= 0 or 2 * c["K"] == n)
    return not (c["K"] <= 0 or 2 * c["K"] == c["nphi"])


def _moves(groups, nphi):
    """Mean number of distinct states one two-body move away (and the state itself); groups: electrons per block."""
    n = 1.0
    for i, a in enumerate(groups):
        n += a * (a - 1) / 2 * ((nphi - a + 2) * (nphi - a + 1) / 2 / nphi - 1)
        for b in groups[i + 1:]:
            n += a * b * ((nphi - a + 1) * (nphi - b + 1) / nphi - 1)
    return max(n, 1.0)


def _size(c):
    """Mean dimension of such a sector and entries of a row."""
    nphi, nel = c["nphi"], c["nel"]
    if c["kind"] == "mono":
        C = math.gcd(nel, nphi)
        return max(1.0, math.comb(nphi, nel) / nphi / C), _moves([nel], nphi)
    if c["kind"] == "spin":
        up, su = c["nel_up"], c["nel_su"]
        tot = sum(math.comb(nphi, a) * math.comb(nphi, up - a) * math.comb(nphi, su - a) *
                  math.comb(nphi, nel - up - su + a) for a in range(max(0, su + up - nel), min(up, su) + 1))
        q = [up * su / nel, up * (nel - su) / nel, (nel - up) * su / nel, (nel - up) * (nel - su) / nel]
        dim = tot / nphi / math.gcd(nel, nphi)
        return max(1.0, dim), min(dim, _moves(q, nphi))
    if c["nel_up"] < 0:
        tot, g = math.comb(2 * nphi, nel), [nel / 2, nel / 2]
    else:
        tot, g = math.comb(nphi, c["nel_up"]) * math.comb(nphi, nel - c["nel_up"]), [c["nel_up"], nel - c["nel_up"]]
    dim = tot / nphi / (math.gcd(nel, nphi) if c.get("K", 0) >= 0 else 1)
    return max(1.0, dim), min(dim, _moves(g, nphi))


def work(case):
    """Bytes and operations of one pass: the CSR written once and read by every product, every stored Krylov vector
    read once per Gram-Schmidt pass, the Ritz vector; MLP: the three GEMMs of each layer and the data read once."""
    c = dict(case)
    if c["kind"] == "mlp":
        dim = _size(dict(c, kind="ground", K=0))[0]
        rows, W, k0 = dim * c["points"], c["width"], (2 * c["nphi"] + 2 + 31) // 32 * 32
        params = k0 * W + 2 * W * W + 4 * W + 1
        return {"bytes": 8.0 * rows + 8.0 * dim + 8.0 * params + 8.0 * dim,
                "flops": 6.0 * rows * (k0 * W + 2 * W * W + W) + 2.0 * dim * (k0 * W + 2 * W * W + W)}
    n = 1
    if c["kind"] == "batch":
        c = dict(c, J=0, K=1, n=c["sectors"] * c["points"])
        n = c["sectors"] * c["points"]
    dim, row = _size(c)
    z = 2 if _complex(c) else 1
    m = min(c["steps"], dim) if not c.get("tol") else min(40, dim)
    vs = (8 if c.get("precision", "f64") == "f64" else 4) * z
    nnz = dim * row
    return {"bytes": n * ((m + 2) * nnz * (4 + vs) + m * (m + 1) / 2 * dim * 8 * z + m * dim * 8 * z),
            "flops": n * z * z * (2 * (m + 2) * nnz + 4 * m * (m + 1) / 2 * dim)}


# ---------------------------------------------------------------------------
# inputs


def _prec(c):
    return B.VAL_FP64 if c["precision"] == "f64" else B.VAL_FP32


def _params(case, seed):
    r = np.random.RandomState(seed % (1 << 31))
    if case["kind"] == "batch":
        ds = np.round(0.2 + 2.6 * r.random_sample(case["points"]), 4)
        return dict(ds=[float(x) for x in ds])
    if case["kind"] == "mono":
        return dict(gamma=float(0.8 + 0.4 * r.random_sample()))
    return dict(d=float(0.4 + 1.6 * r.random_sample()))


def _instances(case, seed):
    p = _params(case, seed)
    return [B.instance(case["nphi"], case["nel"], case["nel_up"], case["J"], K, d)
            for d in p["ds"] for K in range(case["sectors"])]


def _mlp_conds(case):
    return [(3.0 * i / max(1, case["points"] - 1), 0.0) for i in range(case["points"])]


def _mlp_targets(case, seed, dim):
    r = np.random.RandomState(seed % (1 << 31))
    t = r.standard_normal((case["points"], dim)) * np.exp(2.0 * r.random_sample(dim) - 4.0 * r.random_sample(dim))
    return t / np.linalg.norm(t, axis=1, keepdims=True)


def _mlp_weights(case, seed):
    r = np.random.RandomState(seed % (1 << 31) ^ 0x5A5A)
    W, k0 = case["width"], (2 * case["nphi"] + 2 + 31) // 32 * 32
    parts = []
    for fan, shape in ((2 * case["nphi"] + 2, (W, k0)), (W, (W, W)), (W, (W, W))):
        parts += [r.standard_normal(shape).ravel() / math.sqrt(fan), 0.1 * r.standard_normal(W)]
    parts += [r.standard_normal(W) / math.sqrt(W), np.zeros(1)]
    return np.concatenate(parts).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, seed=seed % (1 << 31))
    if kind == "batch":
        s["instances"] = _instances(case, seed)
        return s
    if kind == "mlp":
        basis = B.Basis(case["nphi"], case["nel"], case["nel_up"], 0, 0, rep_mode=B.REP_MIN)
        mlp = B.MLP(2 * case["nphi"], case["width"], seed=1)
        mlp.set_params(_mlp_weights(case, seed))
        s.update(basis=basis, mlp=mlp, conds=_mlp_conds(case), targets=_mlp_targets(case, seed, basis.dim),
                 held_out=float(np.random.RandomState(s["seed"]).uniform(0.1, 2.9)))
        return s
    s.update(_params(case, seed))
    if kind == "ground":
        b = B.Basis(case["nphi"], case["nel"], case["nel_up"], case["J"], case["K"])
        dt = np.complex128 if _complex(case) else np.float64
        s["psi"] = None if case["tol"] else np.zeros(b.dim, dt)  # the caller's buffer for the ground state
        if case["start"]:
            r = np.random.RandomState(s["seed"] ^ 0x1234)
            x = r.random_sample(b.dim) - 0.5
            s["start"] = x + 1j * (r.random_sample(b.dim) - 0.5) if dt == np.complex128 else x
        b.close()
    return s


# ---------------------------------------------------------------------------
# one pass


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "ground":
        r = B.ground_state(c["nphi"], c["nel"], c["nel_up"], c["J"], c["K"], s["d"], c["delta_sas"], c["delta_v"],
                           precision=_prec(c), max_steps=c["steps"], tol=c["tol"], seed=s["seed"],
                           start=s.get("start"), psi_out=s["psi"])
        return dict(energy=np.float64(r["energy"]), ritz0=np.float64(r["ritz0"]), dim=r["dim"], nnz=r["nnz"],
                    steps=r["steps"], psi=r.get("psi"))
    if kind == "spin":
        b = B.basis_spin(c["nphi"], c["nel"], c["nel_up"], c["nel_su"], c["J"], c["K"])
        H = B.hamiltonian_spin(b, s["d"], 0.0, 0.01, 0.02)
        L = B.Lanczos(H, max_steps=c["steps"], tol=c["tol"], seed=s["seed"])
        L.iterate()
        psi = L.ritz_vector()
        out = dict(energy=np.float64(L.rayleigh()), dim=b.dim, nnz=H.nnz, psi=psi)
        o = L.observables_spin(b)  # as one vector: the polarisations vanish in symmetric sectors
        out["observables"] = np.concatenate([[v for k, v in sorted(o.items()) if k != "occupation"],
                                             o["occupation"].ravel()])
        L.close()
        H.close()
        b.close()
        return out
    if kind == "mono":
        r = B.ground_state_mono(c["nphi"], c["nel"], c["J"], c["K"], s["gamma"], max_steps=c["steps"], tol=c["tol"],
                                seed=s["seed"], want_psi=True)
        return dict(energy=np.float64(r["energy"]), level0=r["eigenvalues"], dim=r["dim"], nnz=r["nnz"], psi=r["psi"])
    if kind == "batch":
        b = B.Batch(s["instances"], lam=c["steps"], precision=_prec(c), seed=s["seed"])
        b.solve()
        r = b.results()
        psi = np.concatenate([b.ground_state(i).view(np.float64) for i in range(b.n)])
        b.close()
        return dict(energy=np.array([x["energy"] for x in r]), ritz0=np.array([x["ritz0"] for x in r]),
                    dim=np.array([x["dim"] for x in r]), nnz=np.array([x["nnz"] for x in r]), psi=psi)
    loss, grad = s["mlp"].loss_grad(s["basis"], s["conds"], s["targets"])
    return dict(loss=np.float64(loss), grad=grad, predict=s["mlp"].predict(s["basis"], s["held_out"]))


# ---------------------------------------------------------------------------
# the same results in 64 bits, from the model's definition


def _popcount(x):
    x = x - ((x >> 1) & 0x5555555555555555)
    x = (x & 0x3333333333333333) + ((x >> 2) & 0x3333333333333333)
    x = (x + (x >> 4)) & 0x0F0F0F0F0F0F0F0F
    x = x + (x >> 8)
    x = x + (x >> 16)
    return (x + (x >> 32)) & 0x7F


def _subsets(n, k, dev):
    """All n-bit words with k bits set, ascending."""
    a = torch.zeros(1, dtype=torch.int64, device=dev)
    cnt = torch.zeros(1, dtype=torch.int64, device=dev)
    for b in range(n - 1, -1, -1):
        a, cnt = torch.cat([a, a | (1 << b)]), torch.cat([cnt, cnt + 1])
        ok = (cnt <= k) & (cnt + b >= k)
        a, cnt = a[ok], cnt[ok]
    return a.sort().values


def _rotate(x, bits, nphi, nblocks):
    """Every block rotated left by `bits`, and the parity of the electrons that pass each other."""
    if bits == 0:
        return x, torch.zeros_like(x)
    mask, out, par = (1 << nphi) - 1, torch.zeros_like(x), torch.zeros_like(x)
    for b in range(nblocks):
        y = (x >> (b * nphi)) & mask
        nc = _popcount(y >> (nphi - bits))
        par = par + nc * (_popcount(y) - nc)
        out = out | ((((y << bits) | (y >> (nphi - bits))) & mask) << (b * nphi))
    return out, par & 1


def _tables(nphi, lx, ly, d, mono):
    """Interaction tables V[s][|t|] (within a layer, between layers) and the background energy per electron."""
    i, j = np.meshgrid(np.arange(nphi), np.arange(nphi), indexing="ij")
    off = (i + j) > 0
    if mono:
        z = (i * i * lx / ly + j * j * ly / lx)[off] * np.pi
        ec = (-2.0 + sum(math.sqrt(math.pi / v) * math.erfc(math.sqrt(v)) for v in z)) / math.sqrt(lx * ly)
        ranges = [(np.arange(-(nphi // 2), nphi // 2 + 1), 0.0)]
    else:
        z = (i * i * lx / ly + j * j * ly / lx)[off] * np.pi
        ec = (-2.0 + sum(math.erfc(math.sqrt(v)) for v in z)) / math.sqrt(lx * ly)
        top = 10 * nphi / (d + 0.01)
        ranges = [(np.arange(-nphi, nphi + 1), 0.0), (np.arange(int(-top), math.ceil(top)), d)]
    V = np.zeros((2, nphi, nphi))
    s = np.arange(nphi)
    for a, (qx, dist) in enumerate(ranges):
        for qy in range(nphi):
            x = qx[(qx != 0) | (qy != 0)].astype(np.float64)
            q = np.sqrt(x * x / (lx * lx) + qy * qy / (ly * ly)) * 2 * np.pi
            f = 2 * np.pi / q * np.exp(-q * q / 2 - q * dist)
            V[a, :, qy] = (2 * f[None, :] * np.cos(2 * np.pi * s[:, None] * x[None, :] / nphi)).sum(1) / (2 * lx * ly)
    return V, ec


def _sector_states(m, dev):
    """The states of the orbits that momentum J meets, ascending: T adds nel * q to a state's momentum."""
    nphi = m["nphi"]
    g = math.gcd(m["nel"] * m["q"], nphi) if m["C"] > 1 else nphi
    if m["layers"] is None:
        x = _subsets(m["nblocks"] * nphi, m["nel"], dev)
    else:
        w = m["nblocks"] // 2 * nphi
        lo, hi = _subsets(w, m["layers"][0], dev), _subsets(w, m["layers"][1], dev)
        x = (lo[None, :] | (hi[:, None] << w)).reshape(-1)
    mom = torch.zeros_like(x)
    for o in range(m["nblocks"] * nphi):
        mom += ((x >> o) & 1) * (o % nphi)
    x = x[(mom - m["J"]) % g == 0] if m["J"] >= 0 else x
    if m["spin_up"] is not None:
        mk = (1 << nphi) - 1
        x = x[(_popcount(x & mk) + _popcount((x >> (2 * nphi)) & mk)) == m["spin_up"]]
    return x


def _representatives(m, x):
    """Smallest member of each orbit that carries momentum K, and the orbit's period."""
    C, q = m["C"], m["q"]
    keep = torch.ones_like(x, dtype=torch.bool)
    period = torch.full_like(x, C)
    ok = torch.ones_like(keep)
    for r in range(C - 1, 0, -1):
        y, par = _rotate(x, r * q, m["nphi"], m["nblocks"])
        keep &= y >= x
        same = y == x
        period = torch.where(same, torch.full_like(period, r), period)
        ph = (2 * m["K"] * r + par * C) % (2 * C)  # phase of T^r on the state, in units of pi / C
        ok &= ~same | (ph == 0)
    return x[keep], period[keep], ok[keep]


def _lowest_energy(m):
    """Lowest eigenvalue of the sector's Hamiltonian in the orbit basis (all in 64 bits)."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    nphi, nb, C, q = m["nphi"], m["nblocks"], m["C"], m["q"]
    reps, period, ok = _representatives(m, _sector_states(m, dev))
    reps, period = reps[ok], period[ok]
    n = len(reps)
    prs, trg, amp = [], [], []
    blk = nphi * nb
    ts = range(-(nphi // 2), nphi // 2 + 1) if m["mono"] else range(-(nphi - 1), nphi)
    for a in range(blk):
        for b in range(a + 1, blk):
            ba, bb = a // nphi, b // nphi
            tab = m["V"][0 if (nb == 1 or ba * 2 // nb == bb * 2 // nb) else 1]
            for t in ts:
                a2, b2 = ba * nphi + (a % nphi + t) % nphi, bb * nphi + (b % nphi - t) % nphi
                if a2 != b2:
                    prs.append((a, b))
                    trg.append((a2, b2))
                    amp.append(tab[abs(b2 % nphi - a % nphi), abs(t)])
    N, M = (torch.tensor(v, device=dev) for v in zip(*prs))
    NT, MT = (torch.tensor(v, device=dev) for v in zip(*trg))
    A = torch.tensor(amp, dtype=torch.float64, device=dev)
    rows, cols, vals = [], [], []
    one = torch.ones((), dtype=torch.int64, device=dev)

    def below(x, o):
        return _popcount(x & ((one << o) - 1))

    def add(src, x, h, par):
        best, l, sg = x, torch.zeros_like(x), par
        for r in range(1, C):
            y, p = _rotate(x, r * q, nphi, nb)  # y = T^r x up to sign: x = T^(C - r) y
            less = y < best
            best = torch.where(less, y, best)
            l = torch.where(less, torch.full_like(l, C - r), l)
            sg = torch.where(less, par + p, sg)
        at = torch.searchsorted(reps, best).clamp(max=n - 1)
        hit = reps[at] == best
        src, at, l, sg, h = src[hit], at[hit], l[hit], sg[hit], h[hit]
        v = h * (1 - 2 * (sg & 1)) * torch.sqrt(period[src].double() / period[at].double())
        ang = 2 * math.pi * m["K"] / C * l.double()
        rows.append(at)
        cols.append(src)
        vals.append(torch.complex(v * torch.cos(ang), v * torch.sin(ang)))

    step = max(1, 8_000_000 // len(amp))
    for s0 in range(0, n, step):
        x = reps[s0:s0 + step, None]
        rest = x & ~((one << N) | (one << M))
        hit = ((x >> N) & (x >> M) & 1 & ~(rest >> NT) & ~(rest >> MT)).bool()
        i, k = hit.nonzero(as_tuple=True)
        xi, ni, mi, nt, mt = reps[s0 + i], N[k], M[k], NT[k], MT[k]
        r1 = xi & ~(one << ni)
        r2 = r1 & ~(one << mi)
        r3 = r2 | (one << mt)
        add(s0 + i, r3 | (one << nt), A[k], below(xi, ni) + below(r1, mi) + below(r2, mt) + below(r3, nt))
    if m["tunnel"]:
        everyone = torch.arange(n, device=dev)
        for ba, bb in m["tunnel_blocks"]:
            for o in range(nphi):
                for u, v in ((ba * nphi + o, bb * nphi + o), (bb * nphi + o, ba * nphi + o)):
                    hit = (((reps >> u) & 1) == 1) & (((reps >> v) & 1) == 0)
                    xi = reps[hit]
                    r1 = xi & ~(one << u)
                    add(everyone[hit], r1 | (one << v), torch.full((len(xi),), -0.5 * m["tunnel"], dtype=torch.float64,
                                                                   device=dev), below(xi, u) + below(r1, v))
    mk = (1 << nphi) - 1
    cnt = [_popcount((reps >> (b * nphi)) & mk).double() for b in range(nb)]
    diag = m["diag"](cnt).to(torch.complex128)
    rows.append(torch.arange(n, device=dev))
    cols.append(torch.arange(n, device=dev))
    vals.append(diag)
    H = torch.sparse_coo_tensor(torch.stack([torch.cat(rows), torch.cat(cols)]), torch.cat(vals), (n, n)).coalesce()
    if n <= 1500:
        return np.float64(float(torch.linalg.eigvalsh(H.to_dense())[0]))
    H = H.to_sparse_csr()
    g = torch.Generator().manual_seed(7)
    v = torch.randn(n, 2, generator=g, dtype=torch.float64).to(dev)
    v = torch.view_as_complex(v)
    Q, al, be = [v / torch.linalg.norm(v)], [], []
    for _ in range(min(220, n)):
        w = H @ Q[-1]
        al.append(float(torch.vdot(Q[-1], w).real))
        S = torch.stack(Q)
        for _ in range(2):
            w = w - S.T @ (S.conj() @ w)
        be.append(float(torch.linalg.norm(w)))
        if be[-1] < 1e-10:
            break
        Q.append(w / be[-1])
    return np.float64(np.linalg.eigvalsh(np.diag(al) + np.diag(be[:-1], 1) + np.diag(be[:-1], -1))[0])


def _torus(nphi, gamma=1.0):
    ly = math.sqrt(2 * math.pi * nphi / gamma)
    return ly * gamma, ly


def _model(c, d=None, K=None, gamma=1.0):
    """The sector's Hamiltonian in words: blocks of orbitals, tables, one-body terms."""
    nphi, nel = c["nphi"], c["nel"]
    J, K = c["J"], (c["K"] if K is None else K)
    mono = c["kind"] == "mono"
    lx, ly = _torus(nphi, gamma)
    V, ec = _tables(nphi, lx, ly, d or 0.0, mono)
    m = dict(nphi=nphi, nel=nel, J=J, K=max(K, 0), mono=mono, V=V, tunnel=0.0, spin_up=None, layers=None)
    m["C"] = 1 if K < 0 else (math.gcd(nel, nphi) if mono else nphi)
    m["q"] = nphi // m["C"]
    if mono:
        m.update(nblocks=1, diag=lambda n: ec * nel + 0 * n[0])
    elif c["kind"] == "spin":
        m.update(nblocks=4, layers=(c["nel_up"], nel - c["nel_up"]), spin_up=c["nel_su"],
                 diag=lambda n: ec * nel - d * (n[0] + n[1]) * (n[2] + n[3]) / nphi
                 - 0.5 * 0.01 * (n[0] + n[1] - n[2] - n[3]) - 0.5 * 0.02 * (n[0] + n[2] - n[1] - n[3]))
    else:
        dv = c.get("delta_v", 0.0)
        m.update(nblocks=2, tunnel=c.get("delta_sas", 0.0), tunnel_blocks=((0, 1),),
                 layers=None if c["nel_up"] < 0 else (c["nel_up"], nel - c["nel_up"]),
                 diag=lambda n: ec * nel - d * n[0] * n[1] / nphi + 0.5 * dv * (n[0] - n[1]))
    return m


def _mlp_exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    nphi, W = case["nphi"], case["width"]
    k0 = (2 * nphi + 2 + 31) // 32 * 32
    m = dict(nphi=nphi, nel=case["nel"], J=0, K=0, nblocks=2, C=nphi, q=1, spin_up=None,
             layers=(case["nel_up"], case["nel"] - case["nel_up"]))
    ids = _representatives(m, _sector_states(m, dev))[0]
    dim = len(ids)
    w = torch.tensor(_mlp_weights(case, seed), dtype=torch.float64, device=dev, requires_grad=True)
    parts, o = [], 0
    for shape in ((W, k0), (W,), (W, W), (W,), (W, W), (W,), (W,), (1,)):
        k = int(np.prod(shape))
        parts.append(w[o:o + k].reshape(shape))
        o += k

    def net(d):
        x = torch.zeros(dim, k0, dtype=torch.float64, device=dev)
        for b in range(2 * nphi):
            x[:, b] = (((ids >> b) & 1) * 2 - 1).double()
        x[:, 2 * nphi] = d / 3.0
        for layer in range(3):
            x = torch.tanh(x @ parts[2 * layer].T + parts[2 * layer + 1])
        return x @ parts[6] + parts[7]

    t = torch.tensor(_mlp_targets(case, seed, dim), device=dev)
    loss, grad = 0.0, torch.zeros_like(w)
    for p, (d, _) in enumerate(_mlp_conds(case)):
        out = net(d)
        one = (1 - (out @ t[p]) ** 2 / ((out @ out) * (t[p] @ t[p]))) / case["points"]
        loss += float(one.detach())
        grad += torch.autograd.grad(one, w)[0]
    with torch.no_grad():
        y = net(float(np.random.RandomState(seed % (1 << 31)).uniform(0.1, 2.9)))
        y = y / torch.linalg.norm(y)
    return dict(loss=np.float64(loss), grad=grad.cpu().numpy(), predict=y.cpu().numpy())


def exact(case, seed):
    """Energies of the sectors whose Hamiltonian is built in a few seconds here; a ground state has a free phase and
    is set by the choice of representatives, so it has no value of its own. Odd Nphi bilayers follow a sign rule that
    is no many-body Hamiltonian's, and sectors beyond ~1e5 states take too long."""
    kind = case["kind"]
    p = _params(case, seed)
    if kind == "mlp":
        return _mlp_exact(case, seed)
    if kind == "batch":
        if case["nphi"] > 8 or case["sectors"] * case["points"] > 24:
            return None
        e = [_lowest_energy(_model(case, d, K=K)) for d in p["ds"] for K in range(case["sectors"])]
        return dict(energy=np.array(e), ritz0=np.array(e), dim=None, nnz=None, psi=None)
    if kind == "mono":
        if case["nphi"] > 24:
            return None
    elif case["nphi"] % 2 or _size(case)[0] > (30000 if kind == "spin" else 70000):
        return None
    e = _lowest_energy(_model(case, p.get("d"), gamma=p.get("gamma", 1.0)))
    if kind == "mono":
        return dict(energy=e, level0=np.array([e]), dim=None, nnz=None, psi=None)
    if kind == "spin":
        return dict(energy=e, dim=None, nnz=None, psi=None, observables=None)
    return dict(energy=e, ritz0=e, dim=None, nnz=None, steps=None, psi=None)
