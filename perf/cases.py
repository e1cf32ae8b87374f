"""Workloads of the integral set-up and the SCF step, as a user's program
runs them, for timing and for comparing results.

A case names a path, a cell and a k-point mesh:

  path   build    the four builds of setupSCF (OL, KE, NP, every EP term) of a
                  staged context into device memory, IntegralSetup.build
         graph    the same through build_graph (repeated builds of one context)
         setup    scf.device_integrals: staging, all builds, the context freed:
                  what every SCF run does once per structure
         dropin   the calls of the Fortran boundary: staging and the four
                  builds into host arrays
         ham      the Hamiltonian of a post-SCF run, ham_pscf
         optical  the momentum and dipole matrices of an optical run
         scf      one SCF step on resident integrals: the secular equation's
                  eigensystem, the populations and the valence charge
  cell   si | diamond (conventional cells, `reps` repeated), graphite (AB,
         `reps` repeated), quartz (alpha-SiO2, `reps` repeated), primitive
         (the two-atom diamond cell)
  mesh   a Monkhorst-Pack mesh shifted by 1/2, or "gamma"

Every seed draws its own jittered positions.  Everything is FP64, the only
type the library has.
"""

import math

import numpy as np
import torch

from imago_b200 import charge, configs, intg, scf, secular

# scratch given to a context: a user's program keeps most of the card for its
# matrices
SCRATCH = 24 << 30


def _case(name, path, cell, reps, mesh, spin=1, rel=False):
    return {"name": name, "path": path, "cell": cell, "reps": reps, "mesh": mesh,
            "spin": spin, "rel": rel}


def listed():
    return [
        # the smallest cell a run has, rebuilt: launches and latency
        _case("diamond2_444_graph", "graph", "primitive", "1x1x1", "4x4x4"),
        # a Fortran driver's call on a small supercell: staging, host arrays
        _case("diamond16_222_dropin", "dropin", "diamond", "2x1x1", "2x2x2"),
        # the library's headline benchmark: many k-points, a small cell
        _case("si8_888_build", "build", "si", "1x1x1", "8x8x8"),
        # an ordinary cell with an odd mesh and sizes that fill no tile
        _case("si16_333_build", "build", "si", "2x1x1", "3x3x3"),
        # one cell of the batched stream of 64-atom structures, from scratch
        _case("graphite64_222_setup", "setup", "graphite", "4x4x1", "2x2x2"),
        # the 162-atom quartz supercell at Gamma, real arithmetic
        _case("quartz162_gamma_build", "build", "quartz", "3x3x2", "gamma"),
        # the same with k-points: the largest
        _case("quartz162_222_build", "build", "quartz", "3x3x2", "2x2x2"),
        # the post-SCF Hamiltonian of the headline cell
        _case("si8_888_ham", "ham", "si", "1x1x1", "8x8x8"),
        # ... of a spin-polarised, scalar-relativistic run on a larger cell
        _case("si32_222_ham_spin_rel", "ham", "si", "2x2x1", "2x2x2", 2, True),
        # optical matrices
        _case("si16_444_optical", "optical", "si", "2x1x1", "4x4x4"),
        # an SCF step of the headline cell, and of a small one
        _case("si8_888_scf", "scf", "si", "1x1x1", "8x8x8"),
        _case("diamond16_333_scf", "scf", "diamond", "2x1x1", "3x3x3"),
    ]


# What draw() takes a path's cells from: (cell, repetitions), with the meshes
# that keep a case within the largest listed one.
_SMALL = [("primitive", "1x1x1"), ("diamond", "1x1x1"), ("si", "1x1x1"), ("graphite", "2x1x1"),
          ("quartz", "1x1x1"), ("graphite", "2x2x1"), ("diamond", "2x1x1"), ("si", "2x1x1")]
_LARGE = [("quartz", "2x1x1"), ("si", "2x2x1"), ("diamond", "2x2x1"), ("graphite", "3x2x1"),
          ("quartz", "2x2x1"), ("diamond", "2x2x2"), ("si", "2x2x2"), ("graphite", "4x3x1"),
          ("quartz", "2x2x2"), ("diamond", "3x2x2"), ("graphite", "3x3x2"), ("quartz", "3x2x2")]
_DENSE = ["3x3x3", "4x4x4", "5x5x5", "6x6x6", "4x4x2", "5x4x3", "8x8x2", "7x7x5"]
_COARSE = ["gamma", "2x2x2", "1x1x2", "2x2x1", "3x2x1", "3x2x2"]


def draw(rng):
    path = rng.choice(["build", "build", "build", "graph", "setup", "dropin", "ham", "ham",
                       "optical", "scf"])
    spin, rel = (rng.choice([1, 2]), rng.random() < 0.5) if path == "ham" else (1, False)
    if path == "scf":  # insulators: their filling does not hang on rounding
        cell, reps = rng.choice([c for c in _SMALL if c[0] not in ("graphite", "quartz")])
        mesh = rng.choice(["2x2x2", "3x3x3", "4x4x4", "5x4x3"])
    elif path == "dropin":
        cell, reps = rng.choice(_SMALL)
        mesh = rng.choice(_COARSE)
    elif rng.random() < 0.5:
        cell, reps = rng.choice(_SMALL)
        mesh = rng.choice(_DENSE + _COARSE)
    else:
        cell, reps = rng.choice(_LARGE)
        mesh = rng.choice(_COARSE)
    return {"path": path, "cell": cell, "reps": reps, "mesh": mesh, "spin": spin, "rel": rel}


def _ints(text):
    return tuple(int(x) for x in text.split("x"))


def _system(case, seed):
    reps, gamma = _ints(case["reps"]), case["mesh"] == "gamma"
    k = (1, 1, 1) if gamma else _ints(case["mesh"])
    cell = case["cell"]
    if cell == "primitive":
        s = configs.diamond_primitive(kmesh=k)
        rng = np.random.default_rng(seed)
        pos = s.site_pos + rng.normal(0.0, 0.02 * configs.ANGSTROM, size=s.site_pos.shape)
        s.site_pos = pos
        s.pot_site_pos = pos.copy()
    elif cell == "quartz":
        s = configs.quartz_supercell(reps=reps, kmesh=k, seed=seed, gamma=gamma)
    elif cell == "graphite":
        s = configs.graphite_cell(reps=reps, kmesh=k, seed=seed, jitter=0.02)
    else:
        s = configs.cubic_supercell(cell, reps=reps, kmesh=k, seed=seed, jitter=0.02)
    if gamma:
        s.kpoints_abc = np.zeros((1, 3))
        s.kmesh = None
    return s


def _coeffs(system, spin, seed):
    """Potential coefficients: the atomic start of a run, the second spin's
    a little off; where the data has none (quartz), numbers of that size."""
    try:
        c = scf.atomic_start(system)
    except ValueError:
        c = np.random.default_rng(seed).normal(0.0, 1.0, size=system.pot_dim)
    if spin == 1:
        return c
    d = np.random.default_rng(seed + 1).normal(0.0, 0.01, size=c.shape)
    return np.stack([c * (1.0 + d), c * (1.0 - d)], axis=1)


def _buffers(g):
    f64, dev = torch.float64, torch.device("cuda", 0)
    C = max(g.core_dim, 1)
    shapes = {"ol_packed": (g.nk, g.npacked, 2), "ol_cv_re": (g.nk, g.vale_dim, C),
              "ol_cv_im": (g.nk, g.vale_dim, C), "ke_packed": (g.nk, g.npacked, 2),
              "np_packed": (g.nk, g.npacked, 2), "ep_packed": (g.pot_dim, g.nk, g.npacked, 2)}
    return {k: torch.zeros(v, dtype=f64, device=dev) for k, v in shapes.items()}


def prepare(case, seed):
    path = case["path"]
    system = _system(case, seed)
    state = {"path": path, "system": system}
    if path in ("setup", "dropin"):
        return state
    if path == "scf":
        state["coeffs"] = _coeffs(system, 1, seed)
        state["electrons"] = scf.valence_electrons(system)
        state["integrals"] = scf.device_integrals(system)[0]
        return state
    g = intg.IntegralSetup(system, outputs_on_device=True, scratch_bytes=SCRATCH)
    state["setup"] = g
    if path in ("build", "graph"):
        state["out"] = _buffers(g)
        return state
    # a post-SCF run holds the overlap of the same context
    ol = {k: v for k, v in _buffers(g).items() if k.startswith("ol_")}
    g.build(intg.IMAGO_OL, out=ol)
    if path == "ham":
        state["coeffs"] = _coeffs(system, case["spin"], seed)
        state["rel"] = case["rel"]
        state["out"] = torch.zeros((case["spin"], g.nk, g.npacked, 2), dtype=torch.float64,
                                   device="cuda")
    else:
        state["center"] = system.site_pos.mean(axis=0)
        state["mm"] = torch.zeros((3, g.nk, g.npacked, 2), dtype=torch.float64, device="cuda")
        state["dm"] = torch.zeros_like(state["mm"])
    return state


def run(state):
    path = state["path"]
    if path == "build":
        return state["setup"].build(out=state["out"])
    if path == "graph":
        return state["setup"].build_graph(state["out"])
    if path == "setup":
        return scf.device_integrals(state["system"])[0]
    if path == "dropin":
        with intg.IntegralSetup(state["system"]) as g:
            ol, cv_re, cv_im = g.gauss_overlap_ol()
            return {"ol_packed": ol, "ol_cv_re": cv_re, "ol_cv_im": cv_im,
                    "ke_packed": g.gauss_overlap_ke(), "np_packed": g.gauss_overlap_np(),
                    "ep_packed": g.elec_pot_gauss_overlap()}
    if path == "ham":
        return state["setup"].ham_pscf(state["coeffs"], rel=state["rel"], out=state["out"])
    if path == "optical":
        return {"mm": state["setup"].gauss_overlap_mm(out=state["mm"]),
                "dm": state["setup"].gauss_overlap_dm(state["center"], out=state["dm"])}
    out, w = state["integrals"], state["coeffs"]
    e, c = secular.secular_eigensystem(out, w)
    pop = charge.populate_standard(e.cpu().numpy()[:, None, :], state["electrons"])
    r = charge.valence_rho(out, [e], [c], pop["population"], w)
    # the vectors themselves are defined up to phases and rotations of
    # degenerate levels; what the step hands on is their density
    return {"eigenvalues": e, "density": charge.packed_density(c, pop["population"][:, 0, :]),
            "fermi": pop["occupied_energy"], "potRho": r["potRho"],
            "kinetic": r["kineticEnergyTrace"], "nuclear": r["nucPotTrace"],
            "charge": r["chargeDensityTrace"], "electronEnergy": r["electronEnergy"]}


# ------------------------------------------------------------------ work --
def work(case):
    s = _system(case, 1)
    V, C, nk, P = s.vale_dim, s.core_dim, s.num_kpoints, s.pot_dim
    npk = V * (V + 1) // 2
    packed = 16.0 * nk * npk
    path = case["path"]
    if path == "scf":
        occ = scf.valence_electrons(s) / 2.0
        return {"bytes": packed * (P + 4) + 8.0 * nk * V,
                # Cholesky, the reduction, a full eigensystem (reduction to
                # tridiagonal, vectors back), the density, the traces
                "flops": nk * (V ** 3 * (4 / 3 + 8 + 16 / 3 + 16) + 8 * occ * npk)
                + 4.0 * nk * npk * (P + 3)}
    T = -math.log(s.basis_fn_convg)
    omega = abs(np.linalg.det(s.real_vectors))
    counts = np.bincount(s.site_type, minlength=len(s.atom_types) + 1)[1:]
    pots = np.bincount(s.pot_site_type, minlength=len(s.pot_types) + 1)[1:]
    pair_flops = {"ol": 0.0, "ep": 0.0, "np": 0.0, "contract": 0.0, "phase": 0.0}
    for i, ti in enumerate(s.atom_types):
        for j, tj in enumerate(s.atom_types):
            a, b = ti.alphas[:, None], tj.alphas[None, :]
            la = np.array([max(q for q in range(4) if n < ti.num_orb_alphas[q])
                           for n in range(len(ti.alphas))])[:, None]
            lb = np.array([max(q for q in range(4) if n < tj.num_orb_alphas[q])
                           for n in range(len(tj.alphas))])[None, :]
            xi, zeta, L = a * b / (a + b), a + b, la + lb
            sph = ((la + 1) * (lb + 1)) ** 2
            herm = (L + 1) * (L + 2) * (L + 3) / 6
            half = 0.5 * counts[i] * counts[j]
            rows = half * 4 / 3 * math.pi * (T / xi) ** 1.5 / omega
            n_i = ti.num_vale_states + ti.num_core_states
            n_j = tj.num_vale_states + tj.num_core_states
            pair_flops["ol"] += (rows * 6 * sph).sum()
            pair_flops["contract"] += (rows * 2 * (la + 1) ** 2 * n_j).sum()
            pair_flops["phase"] += half * 4 / 3 * math.pi * (T / xi.min()) ** 1.5 / omega \
                * 4 * n_i * n_j
            for q, p in enumerate(s.pot_types):
                for c in p.alphas:
                    mu = zeta * c / (zeta + c)
                    trip = half * pots[q] * math.pi ** 3 * T ** 3 / (6 * (xi * mu) ** 1.5) \
                        / omega ** 2
                    pair_flops["ep"] += (trip * (30 + 3 * herm) + rows * 4 * sph).sum()
                mu = zeta * p.nuc_alpha / (zeta + p.nuc_alpha)
                trip = half * pots[q] * math.pi ** 3 * T ** 3 / (6 * (xi * mu) ** 1.5) / omega ** 2
                pair_flops["np"] += (trip * (60 + 5 * herm) + rows * 2 * sph).sum()
    # H(-k) = conj H(k): half the phase sums and orthogonalisations
    gamma = case["mesh"] == "gamma"
    kk = 0.25 if gamma else (nk + 1) // 2
    per = kk * (8.0 * C * C * V + 16.0 * C * npk) + kk * pair_flops["phase"] \
        + pair_flops["contract"]
    cv = 16.0 * nk * V * C
    if path == "ham":
        n = case["spin"]
        return {"bytes": packed * n + cv,
                "flops": n * per + pair_flops["ep"] + pair_flops["np"] + 2 * pair_flops["ol"]}
    if path == "optical":
        return {"bytes": 6 * packed + cv, "flops": 6 * (per + pair_flops["ol"])}
    return {"bytes": packed * (3 + P) + cv,
            "flops": (3 + P) * per + pair_flops["ep"] + pair_flops["np"] + 2 * pair_flops["ol"]}


# ----------------------------------------------------------------- exact --
# The same integrals and matrices in plain torch: every primitive pair and
# triple whose Gaussian product factor exceeds exp(-_CUT), one-dimensional
# overlap tables, Hermite expansions for the Coulomb term, contraction,
# phase sums and the orthogonalisation to the core, without any of the
# library's code.
_CUT = 44.0
_ANG = [0.2820947917738782] + [0.4886025119029199] * 3 + [1.0925484305920790] * 3 + \
    [0.5462742152960396, 0.3153915652525200]
_CART = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (2, 0, 0), (0, 2, 0), (0, 0, 2),
         (1, 1, 0), (1, 0, 1), (0, 1, 1)]
_SPH = [[(0, 1)], [(1, 1)], [(2, 1)], [(3, 1)], [(7, 1)], [(8, 1)], [(9, 1)],
        [(4, 1), (5, -1)], [(6, 2), (4, -1), (5, -1)]]


def _dev(x):
    return torch.as_tensor(np.ascontiguousarray(x), device="cuda")


class _Exact:
    """The primitive rows (pair, image, alpha 1, alpha 2) of one system."""

    def __init__(self, s):
        self.s = s
        self.lmax = max(max(t.core_l + t.vale_l) for t in s.atom_types)
        rv = np.asarray(s.real_vectors)
        pos, st = s.site_pos, np.asarray(s.site_type) - 1
        self.nst = max(t.num_vale_states + t.num_core_states for t in s.atom_types)
        coef, lm = [], np.zeros((len(s.atom_types), self.nst), np.int64)
        na = max(len(t.alphas) for t in s.atom_types)
        for q, t in enumerate(s.atom_types):
            m, c = 0, np.zeros((na, self.nst))
            for l, f in list(zip(t.vale_l, t.vale_coeffs)) + list(zip(t.core_l, t.core_coeffs)):
                for h in range(l * l, (l + 1) ** 2):
                    lm[q, m] = h
                    c[:len(f), m] = np.asarray(f) * _ANG[h]
                    m += 1
            coef.append(c)
        self.coef, self.lm = _dev(np.stack(coef)), _dev(lm)
        amin = min(t.alphas[0] for t in s.atom_types)
        inv = np.linalg.inv(rv)
        self.pairs = [(i, j) for i in range(len(pos)) for j in range(i, len(pos))]
        ij = np.array(self.pairs)
        d = pos[ij[:, 0]] - pos[ij[:, 1]]
        reach = math.sqrt(_CUT * 2.0 / amin)
        lat = self.lattice(reach + np.abs(rv).sum())
        shift = -np.rint(d @ inv) @ rv               # nearest cell of each pair
        u_pair, u_lat = [], []
        for p in range(len(ij)):
            x = d[p] - (lat - shift[p])
            keep = np.flatnonzero((x * x).sum(1) <= reach * reach)
            u_pair.append(np.full(len(keep), p))
            u_lat.append(lat[keep] - shift[p])
        self.u_pair, self.u_lat = np.concatenate(u_pair), np.concatenate(u_lat)
        A = pos[ij[self.u_pair, 0]]
        B = pos[ij[self.u_pair, 1]] + self.u_lat
        ti, tj = st[ij[self.u_pair, 0]], st[ij[self.u_pair, 1]]
        alph = np.zeros((len(s.atom_types), na))
        for q, t in enumerate(s.atom_types):
            alph[q, :len(t.alphas)] = t.alphas
        alph, A, B, ti, tj = _dev(alph), _dev(A), _dev(B), _dev(ti), _dev(tj)
        a, b = alph[ti][:, :, None], alph[tj][:, None, :]
        xi = a * b / (a + b).clamp(min=1e-300)
        r2 = ((A - B) ** 2).sum(1)[:, None, None]
        u, ia, ib = torch.nonzero((xi * r2 <= _CUT) & (a > 0) & (b > 0), as_tuple=True)
        self.u, self.A, self.B = u, A[u], B[u]
        self.a, self.b = alph[ti[u], ia], alph[tj[u], ib]
        self.c1, self.c2 = self.coef[ti[u], ia], self.coef[tj[u], ib]
        self.lm1, self.lm2 = self.lm[ti], self.lm[tj]  # per unit
        self.zeta = self.a + self.b
        self.P = (self.a[:, None] * self.A + self.b[:, None] * self.B) / self.zeta[:, None]
        self.e0 = self.a * self.b / self.zeta * ((self.A - self.B) ** 2).sum(1)
        self.kxyz = np.asarray(s.kpoints_abc) @ (2 * math.pi * inv.T)
        ph = np.exp(1j * (self.u_lat @ self.kxyz.T))
        self.phase = _dev(ph)                        # [unit, k]

    def lattice(self, radius):
        rv = np.asarray(self.s.real_vectors)
        n = [int(radius * np.linalg.norm(np.linalg.inv(rv)[:, i])) + 1 for i in range(3)]
        g = np.stack(np.meshgrid(*[np.arange(-m, m + 1) for m in n], indexing="ij"), -1)
        lat = g.reshape(-1, 3) @ rv
        return lat[(lat * lat).sum(1) <= radius * radius]

    def table(self, PA, PB, p, na, nb):
        """1D overlap tables S[i][j], S00 = 1; inputs [rows, 3]."""
        h = 0.5 / p[:, None]
        S = [[None] * (nb + 1) for _ in range(na + 1)]
        S[0][0] = torch.ones_like(PA)
        for i in range(na):
            S[i + 1][0] = PA * S[i][0] + (i * h * S[i - 1][0] if i else 0.0)
        for j in range(nb):
            for i in range(na + 1):
                S[i][j + 1] = PB * S[i][j] + (i * h * S[i - 1][j] if i else 0.0) \
                    + (j * h * S[i][j - 1] if j else 0.0)
        return S

    def spherical(self, cart):
        """[rows, ns, ns] from a function of two Cartesian indices."""
        ns = (self.lmax + 1) ** 2
        rows = []
        for x in range(ns):
            row = []
            for y in range(ns):
                row.append(sum(c1 * c2 * cart(p, q) for p, c1 in _SPH[x] for q, c2 in _SPH[y]))
            rows.append(torch.stack(row, -1))
        return torch.stack(rows, -2)

    def two(self, op, axis=0, center=None):
        l = self.lmax
        S = self.table(self.P - self.A, self.P - self.B, self.zeta, l + 2, l + 2)
        a, b = self.a[:, None], self.b[:, None]

        def second(i, j):
            return (j * (j - 1) * S[i][j - 2] if j > 1 else 0.0) - 2 * b * (2 * j + 1) * S[i][j] \
                + 4 * b * b * S[i][j + 2]

        def second_both(i, j):
            v = -2 * a * (2 * i + 1) * second(i, j) + 4 * a * a * second(i + 2, j)
            return v + (i * (i - 1) * second(i - 2, j) if i > 1 else 0.0)

        def second_left(i, j):
            return (i * (i - 1) * S[i - 2][j] if i > 1 else 0.0) \
                - 2 * a * (2 * i + 1) * S[i][j] + 4 * a * a * S[i + 2][j]

        def vec(i, j):
            if op == "dm":
                return S[i][j + 1] + (self.B - center) * S[i][j]
            # d/dx on the smaller exponent's side, where nothing cancels
            left = 2 * a * S[i + 1][j] - (i * S[i - 1][j] if i else 0.0)
            right = (j * S[i][j - 1] if j else 0.0) - 2 * b * S[i][j + 1]
            return torch.where(a <= b, left, right)

        pre = (math.pi / self.zeta) ** 1.5 * torch.exp(-self.e0)

        def cart(p, q):
            i, j = _CART[p], _CART[q]
            f = [S[i[x]][j[x]][:, x] for x in range(3)]
            if op == "ol":
                v = f[0] * f[1] * f[2]
            elif op == "ke":
                d = [second(i[x], j[x])[:, x] for x in range(3)]
                v = -0.5 * (d[0] * f[1] * f[2] + f[0] * d[1] * f[2] + f[0] * f[1] * d[2])
            elif op == "mv":
                u = [second_both(i[x], j[x])[:, x] for x in range(3)]
                L = [second_left(i[x], j[x])[:, x] for x in range(3)]
                R = [second(i[x], j[x])[:, x] for x in range(3)]
                v = u[0] * f[1] * f[2] + f[0] * u[1] * f[2] + f[0] * f[1] * u[2]
                v = v + (L[0] * R[1] + R[0] * L[1]) * f[2] + (L[0] * R[2] + R[0] * L[2]) * f[1] \
                    + (L[1] * R[2] + R[1] * L[2]) * f[0]
                v = v * -((7.2973525693e-3) ** 2 / 8)
            else:
                f[axis] = vec(i[axis], j[axis])[:, axis]
                v = f[0] * f[1] * f[2]
            return pre * v
        return self.spherical(cart)

    def three(self, sites, c, z=None):
        """sum over the images of `sites` of exp(-c r^2) (z None) or of
        -z exp(-c r^2) / r, per row, [rows, ns, ns]."""
        L = 2 * self.lmax
        herm = [(t, u, n - t - u) for n in range(L + 1) for t in range(n, -1, -1)
                for u in range(n - t, -1, -1)]
        at = {h: i for i, h in enumerate(herm)}
        mu = self.zeta * c / (self.zeta + c)
        reach = math.sqrt(float(((_CUT - self.e0).clamp(min=0) / mu).max()))
        lo, hi = self.P.min(0).values.cpu().numpy(), self.P.max(0).values.cpu().numpy()
        lat = self.lattice(reach + np.linalg.norm(hi - lo) + np.abs(sites).max() * 2
                           + np.linalg.norm(self.s.real_vectors, axis=1).sum())
        pts = (lat[:, None, :] + sites[None]).reshape(-1, 3)
        pts = _dev(pts[((pts >= lo - reach) & (pts <= hi + reach)).all(1)])
        Q = torch.zeros((len(self.a), len(herm)), dtype=torch.float64, device="cuda")
        chunk = max(1, int(1.5e8) // max(1, len(pts)))
        for r0 in range(0, len(self.a), chunk):
            sl = slice(r0, r0 + chunk)
            d2 = torch.zeros((len(self.a[sl]), len(pts)), dtype=torch.float64, device="cuda")
            for x in range(3):
                d2 += (self.P[sl, x, None] - pts[None, :, x]) ** 2
            r, t = torch.nonzero(mu[sl, None] * d2 + self.e0[sl, None] <= _CUT, as_tuple=True)
            del d2
            for q0 in range(0, len(r), 4_000_000):
                rr, tt = r[q0:q0 + 4_000_000] + r0, t[q0:q0 + 4_000_000]
                X, m = self.P[rr] - pts[tt], mu[rr]
                Q.index_add_(0, rr, self.coulomb(X, m, c, z, rr, herm, at) if z is not None
                             else self.gauss(X, m, herm))
        if z is None:
            pre = (math.pi / (self.zeta + c)) ** 1.5 * torch.exp(-self.e0)
        else:
            pre = torch.exp(-self.e0)
        PA, PB, h = self.P - self.A, self.P - self.B, 0.5 / self.zeta[:, None]
        E = {(0, 0): [torch.ones_like(PA)]}

        def raise_(e, X):
            n = len(e)
            return [(h * e[t - 1] if t > 0 else 0.0) + (X * e[t] if t < n else 0.0)
                    + ((t + 1) * e[t + 1] if t + 1 < n else 0.0) for t in range(n + 1)]
        for i in range(self.lmax + 1):
            if i:
                E[i, 0] = raise_(E[i - 1, 0], PA)
            for j in range(self.lmax):
                E[i, j + 1] = raise_(E[i, j], PB)

        def cart(p, q):
            i, j = _CART[p], _CART[q]
            v = 0.0
            for t, et in enumerate(E[i[0], j[0]]):
                for u, eu in enumerate(E[i[1], j[1]]):
                    for w, ew in enumerate(E[i[2], j[2]]):
                        v = v + et[:, 0] * eu[:, 1] * ew[:, 2] * Q[:, at[t, u, w]]
            return pre * v
        return self.spherical(cart)

    def gauss(self, X, m, herm):
        n = 2 * self.lmax
        h = [torch.ones_like(X)]
        for t in range(n):
            h.append(-2 * m[:, None] * (X * h[t] + (t * h[t - 1] if t else 0.0)))
        g = torch.exp(-m * (X * X).sum(1))
        return torch.stack([g * h[t][:, 0] * h[u][:, 1] * h[v][:, 2] for t, u, v in herm], 1)

    def coulomb(self, X, m, c, z, rr, herm, at):
        n = 2 * self.lmax
        z3 = self.zeta[rr] + c
        nu = self.zeta[rr] ** 2 / z3
        x2 = (X * X).sum(1)
        T = nu * x2
        F = []
        for k in range(n + 1):
            g = math.gamma(k + 0.5)
            big = T > 1e-3
            Tb = torch.where(big, T, torch.ones_like(T))
            f = 0.5 * g * torch.special.gammainc(torch.full_like(Tb, k + 0.5), Tb) / Tb ** (k + 0.5)
            small = sum((-T) ** i / (math.factorial(i) * (2 * k + 2 * i + 1)) for i in range(6))
            F.append(torch.where(big, f, small))
        w = -z * 2 * math.pi / z3 * torch.exp(-m * x2)
        R = [{(0, 0, 0): w * (-2.0) ** k * sum(math.comb(k, i) * m ** (k - i) * nu ** i * F[i]
                                               for i in range(k + 1))} for k in range(n + 1)]
        for h in herm[1:]:
            x = next(q for q in range(3) if h[q])
            one = tuple(h[q] - (q == x) for q in range(3))
            two = tuple(h[q] - 2 * (q == x) for q in range(3))
            for k in range(n + 1 - sum(h)):
                v = X[:, x] * R[k + 1][one]
                R[k][h] = v + ((h[x] - 1) * R[k + 1][two] if h[x] > 1 else 0.0)
        return torch.stack([R[0][h] for h in herm], 1)

    def blocks(self, sh):
        """Contracted [unit, n_i, n_j] blocks of the rows' [ns, ns] ones."""
        M = torch.zeros((len(self.u_pair), self.nst, self.nst), dtype=torch.float64,
                        device="cuda")
        for r0 in range(0, len(self.u), 100_000):
            sl = slice(r0, r0 + 100_000)
            u = self.u[sl]
            x = torch.gather(sh[sl], 1, self.lm1[u][:, :, None].expand(-1, -1, sh.shape[2]))
            x = torch.gather(x, 2, self.lm2[u][:, None, :].expand(-1, self.nst, -1))
            M.index_add_(0, u, x * self.c1[sl][:, :, None] * self.c2[sl][:, None, :])
        return M

    def summed(self, M, factor=1.0):
        """(vv, cv, cc) [k, ...]: the phase sums, each pair's block stored
        as the reference stores it."""
        s = self.s
        V, C, nk = s.vale_dim, s.core_dim, s.num_kpoints
        z = dict(dtype=torch.complex128, device="cuda")
        vv, cv, cc = torch.zeros((nk, V, V), **z), torch.zeros((nk, C, V), **z), \
            torch.zeros((nk, C, C), **z)
        st = np.asarray(s.site_type) - 1
        nv = [s.atom_types[t].num_vale_states for t in st]
        nc = [s.atom_types[t].num_core_states for t in st]
        ov, oc = np.concatenate([[0], np.cumsum(nv)]), np.concatenate([[0], np.cumsum(nc)])
        ends = np.searchsorted(self.u_pair, np.arange(len(self.pairs) + 1))
        for p, (i, j) in enumerate(self.pairs):
            u = slice(ends[p], ends[p + 1])
            b = factor * (self.phase[u].T @ M[u].reshape(-1, self.nst ** 2).to(torch.complex128))
            b = b.reshape(nk, self.nst, self.nst)
            vi, vj = slice(ov[i], ov[i + 1]), slice(ov[j], ov[j + 1])
            ci, cj = slice(oc[i], oc[i + 1]), slice(oc[j], oc[j + 1])
            vale_i, vale_j = slice(0, nv[i]), slice(0, nv[j])
            core_i, core_j = slice(nv[i], nv[i] + nc[i]), slice(nv[j], nv[j] + nc[j])
            vv[:, vi, vj] = b[:, vale_i, vale_j]
            if i != j:
                cv[:, ci, vj] = b[:, core_i, vale_j]
                cc[:, cj, ci] = b[:, core_i, core_j].mH
            cv[:, cj, vi] = b[:, vale_i, core_j].mH
            cc[:, ci, cj] = b[:, core_i, core_j]
        return vv, cv, cc

    def packed(self, parts, S, hermitian=True):
        vv, cv, cc = parts
        V, C = self.s.vale_dim, self.s.core_dim
        col = torch.cat([torch.full((q + 1,), q) for q in range(V)]).cuda()
        row = torch.cat([torch.arange(q + 1) for q in range(V)]).cuda()
        if C:
            w = vv - S.mH @ cv - cv.mH @ S
            d = torch.arange(V, device="cuda")
            w[:, d, d] = w[:, d, d].real.to(w.dtype)
            w = w + S.mH @ cc @ S
            if hermitian:
                w[:, d, d] = w[:, d, d].real.to(w.dtype)
            out = torch.view_as_real(w[:, row, col]).clone()
            out[out.abs() < 1e-10] = 0.0
        else:
            out = torch.view_as_real(vv[:, row, col]).clone()
        return out

    def one(self, sh, S=None, factor=1.0, hermitian=True):
        parts = self.summed(self.blocks(sh), factor)
        return self.packed(parts, parts[1] if S is None else S, hermitian), parts[1]

    def nuclear(self):
        s, pt = self.s, np.asarray(self.s.pot_site_type)
        return sum(self.three(s.pot_site_pos[pt == q + 1], p.nuc_alpha, p.nuc_charge)
                   for q, p in enumerate(s.pot_types))

    def terms(self):
        s, pt = self.s, np.asarray(self.s.pot_site_type)
        for q, p in enumerate(s.pot_types):
            for c in p.alphas:
                yield self.three(s.pot_site_pos[pt == q + 1], float(c))


def _exact_integrals(s):
    x = _Exact(s)
    ol, S = x.one(x.two("ol"))
    cv = S.transpose(1, 2)
    return {"ol_packed": ol, "ol_cv_re": cv.real.contiguous(), "ol_cv_im": cv.imag.contiguous(),
            "ke_packed": x.one(x.two("ke"), S)[0], "np_packed": x.one(x.nuclear(), S)[0],
            "ep_packed": torch.stack([x.one(t, S)[0] for t in x.terms()])}


def _exact_scf(s, w):
    out = _exact_integrals(s)
    V, nk = s.vale_dim, s.num_kpoints
    col = torch.cat([torch.full((q + 1,), q) for q in range(V)]).cuda()
    row = torch.cat([torch.arange(q + 1) for q in range(V)]).cuda()

    def full(p):
        m = torch.zeros((nk, V, V), dtype=torch.complex128, device="cuda")
        m[:, row, col] = torch.view_as_complex(p.contiguous())
        m[:, col, row] = m[:, row, col].conj()
        return m
    f = [1.0 if x == 0.0 else float(x) for x in w]
    h = out["np_packed"] + out["ke_packed"]
    for x, e in zip(f, out["ep_packed"]):
        h = h + x * e
    lo = torch.linalg.cholesky(full(out["ol_packed"]))
    a = torch.linalg.solve_triangular(lo, full(h), upper=False)
    a = torch.linalg.solve_triangular(lo, a.mH, upper=False)
    a = (0.5 * (a + a.mH)).cpu()
    e, y = torch.linalg.eigh(a)
    c = torch.linalg.solve_triangular(lo.mH, y.cuda(), upper=True)
    flat = e.reshape(-1).numpy()
    each = 2.0 / nk
    order, left = np.argsort(flat, kind="stable"), scf.valence_electrons(s)
    pop = np.zeros_like(flat)
    full_states = int(left / each + 1e-9)
    pop[order[:full_states]] = each
    rest = left - full_states * each
    top = full_states - 1
    if rest > 1e-9:
        pop[order[full_states]] = rest
        top = full_states
    pop = torch.as_tensor(pop.reshape(nk, V), device="cuda")
    rho = (c * pop[:, None, :]) @ c.mH
    packed = torch.view_as_real(rho[:, row, col]).clone()
    packed[:, row == col, 1] = 0.0
    weight = torch.where(row == col, 1.0, 2.0).to(torch.float64)[None, :, None]

    def trace(m):
        return float((m * packed * weight).sum())
    return {"eigenvalues": e, "density": packed, "fermi": float(flat[order[top]]),
            "potRho": np.array([[trace(m)] for m in out["ep_packed"]]),
            "kinetic": np.array([trace(out["ke_packed"])]),
            "nuclear": np.array([trace(out["np_packed"])]),
            "charge": np.array([trace(out["ol_packed"])]),
            "electronEnergy": np.array([float((pop.cpu().numpy() * e.numpy()).sum())])}


def exact(case, seed):
    s = _system(case, seed)
    # the plain sums over many atoms or many terms would take minutes
    if len(s.site_pos) > 16 or (case["cell"] == "quartz" and s.num_kpoints > 8):
        return None
    path = case["path"]
    if path == "scf":
        return _exact_scf(s, _coeffs(s, 1, seed))
    if path in ("build", "graph", "setup", "dropin"):
        return _exact_integrals(s)
    x = _Exact(s)
    S = x.one(x.two("ol"))[1]
    if path == "ham":
        c = np.asarray(_coeffs(s, case["spin"], seed)).reshape(s.pot_dim, -1)
        sh = x.two("ke") + x.nuclear() + (x.two("mv") if case["rel"] else 0.0)
        spins = [sh.clone() for _ in range(case["spin"])]
        for t, e in enumerate(x.terms()):
            for q in range(case["spin"]):
                spins[q] += float(c[t, q]) * e
        return torch.stack([x.one(q, S)[0] for q in spins])
    center = _dev(s.site_pos.mean(axis=0))
    return {"mm": torch.stack([x.one(x.two("mm", a), S, -1j)[0] for a in range(3)]),
            "dm": torch.stack([x.one(x.two("dm", a, center), S, 1.0, False)[0]
                               for a in range(3)])}
