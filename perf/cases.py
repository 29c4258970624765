"""The work that users have this framework do, as cases that can be timed and
compared: field evaluation, charge solves, axial tables, electron tracing and
surrogate training, through the public entry points.

A case is a dict of plain values; `kind` names the entry point, the other
keys are its sizes and options.  Inputs are made from the seed alone: the
charges that a field case starts from come from a plain dense solve in this
file, not from the framework's solver.
"""
import math

import numpy as np
import torch

MM = 1e-3
MU0 = 1.25663706212e-06
EVAL_FLOPS = 110592      # one surrogate network evaluation: 2 (16 128 + 3 128^2 + 128 32)
ATTEMPTS = 73            # step attempts of a lens electron at atol 1e-10 (RKF45, six field evaluations each)
RING_FLOPS = 87          # algorithmic flops of one ring's field at one point


def listed():
    return [
        # The field at one point, as a script or notebook asks for it: latency.
        {'name': 'point', 'kind': 'point', 'n_el': 1000},
        # The field of a finely meshed lens on a large point set (2^18 points): the precision workload.
        {'name': 'map_large', 'kind': 'map', 'n_el': 16384, 'points': 1 << 18, 'magnetic': False},
        # An H-field map of a pole piece and its coils, ragged sizes: plotting and tolerancing.
        {'name': 'map_magnetic', 'kind': 'map', 'n_el': 1537, 'points': 9797, 'magnetic': True},
        # A whole charge solve of a magnetizable pole piece in its coils' field (flux rows), ordinary size.
        {'name': 'solve_magnetic', 'kind': 'solve_magnetic', 'n_el': 2501},
        # Eight voltage settings on the finest lens mesh: the precision solve.
        {'name': 'solve_large', 'kind': 'solve', 'n_el': 16384, 'nrhs': 8},
        # A design sweep: eight lens stacks of uneven size solved and traced in one replay.
        {'name': 'sweep', 'kind': 'sweep', 'lenses': 8, 'n_max': 3000, 'electrons': 128},
        # The axial interpolation table of a lens on the 5 um grid used for tracing.
        {'name': 'axial_table', 'kind': 'axial', 'n_el': 1000, 'nz': 4601},
        # A beam through an axial field, host arrays in and out.
        {'name': 'trace_axial', 'kind': 'trace_axial', 'n_el': 1000, 'nz': 4601, 'electrons': 65537, 'log_atol': -10},
        # A beam through the direct BEM field of the lens: the plain method.
        {'name': 'trace_bem', 'kind': 'trace_bem', 'n_el': 1000, 'electrons': 4096, 'log_atol': -10},
        # One electron through a combined electrostatic and magnetic lens.
        {'name': 'trace_single', 'kind': 'trace_single', 'n_el': 1001},
        # A batch of the learned-surrogate beam through its session, end to end.
        {'name': 'trace_surrogate', 'kind': 'trace_surrogate', 'n_el': 1000, 'electrons': 262144},
        # One optimiser step of the surrogate's training.
        {'name': 'train_step', 'kind': 'train', 'batch': 8192, 'n_src': 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['point', 'map', 'solve', 'solve_magnetic', 'sweep', 'axial', 'trace_axial', 'trace_bem',
                       'trace_single', 'trace_surrogate', 'train'])
    if kind == 'point':
        return {'kind': kind, 'n_el': _log(rng, 100, 16384)}
    if kind == 'map':
        return {'kind': kind, 'n_el': _log(rng, 100, 16384), 'points': _log(rng, 16, 1 << 18),
                'magnetic': rng.random() < 0.4}
    if kind == 'solve':
        return {'kind': kind, 'n_el': _log(rng, 100, 16384), 'nrhs': rng.randint(1, 8)}
    if kind == 'solve_magnetic':
        return {'kind': kind, 'n_el': _log(rng, 100, 8192)}
    if kind == 'sweep':
        return {'kind': kind, 'lenses': rng.randint(2, 8), 'n_max': _log(rng, 600, 3000),
                'electrons': _log(rng, 8, 128)}
    if kind == 'axial':
        return {'kind': kind, 'n_el': _log(rng, 100, 16384), 'nz': _log(rng, 51, 4601)}
    if kind == 'trace_axial':
        return {'kind': kind, 'n_el': _log(rng, 200, 1000), 'nz': _log(rng, 1001, 4601),
                'electrons': _log(rng, 1, 65537), 'log_atol': rng.choice([-10, -9, -8])}
    if kind == 'trace_bem':
        return {'kind': kind, 'n_el': _log(rng, 200, 1000), 'electrons': _log(rng, 1, 4096),
                'log_atol': rng.choice([-10, -9, -8])}
    if kind == 'trace_single':
        return {'kind': kind, 'n_el': _log(rng, 200, 3000)}
    if kind == 'trace_surrogate':
        return {'kind': kind, 'n_el': _log(rng, 200, 1000), 'electrons': _log(rng, 100, 262144)}
    return {'kind': kind, 'batch': _log(rng, 256, 8192), 'n_src': rng.randint(1, 7)}


# ---------------------------------------------------------------- plain 64-bit mathematics
def _dev():
    return torch.device('cuda' if torch.cuda.is_available() else 'cpu')


def _elliptic(t):
    """K and E of the complementary parameter t = 1 - k^2, by the arithmetic-geometric mean."""
    a, g = torch.ones_like(t), torch.sqrt(t)
    s, f = 0.5 * (1.0 - t), 1.0
    for _ in range(7):
        c = 0.5 * (a - g)
        a, g = 0.5 * (a + g), torch.sqrt(a * g)
        s = s + f * c * c
        f *= 2.0
    K = (0.5 * math.pi) / a
    return K, K * (1.0 - s)


def _ring(r0, z0, rs, zs, want):
    """'pot', or ('field') E_r and E_z, of unit rings (rs, zs) at (r0, z0); the arguments broadcast."""
    dr, dz = rs - r0, zs - z0
    rho2 = dr * dr + dz * dz
    D = rho2 + 4.0 * r0 * rs
    K, E = _elliptic(rho2 / D)
    q = rs / (math.pi * torch.sqrt(D))
    if want == 'pot':
        return q * K
    er = q * (rho2 * (K - E) - 2.0 * r0 * dr * E) / (2.0 * r0 * rho2)
    return er, -q * dz * E / rho2


def _coil(r0, z0, a, zs):
    """H_r, H_z of a unit current loop of radius a at height zs."""
    z = z0 - zs
    A, B = z * z + (a + r0) ** 2, z * z + (r0 - a) ** 2
    K, E = _elliptic(B / A)
    hr = z / (2 * math.pi * r0 * torch.sqrt(A)) * ((z * z + r0 * r0 + a * a) / B * E - K)
    hz = 1 / (2 * math.pi * torch.sqrt(A)) * ((a * a - z * z - r0 * r0) / B * E + K)
    return hr, hz


class _Elements:
    """Cubic elements (N, 4, 3) = [start, end, 1/3, 2/3]: Gauss rings, collocation points, normals."""

    def __init__(self, vertices):
        v = torch.as_tensor(np.ascontiguousarray(vertices), dtype=torch.float64, device=_dev())
        x0, x3, x1, x2 = (v[:, i][:, [0, 2]] for i in range(4))
        self.k = [(-x3 + 9 * x2 + 9 * x1 - x0) / 16, (-x3 + 27 * x2 - 27 * x1 + x0) / 16,
                  (9 * x3 - 9 * x2 - 9 * x1 + 9 * x0) / 16, (9 * x3 - 27 * x2 + 27 * x1 - 9 * x0) / 16]
        self.n = len(v)
        x, w = np.polynomial.legendre.leggauss(16)
        self.pos, j = self.at(torch.as_tensor(x, device=v.device), False)
        self.jac = torch.as_tensor(w, device=v.device) * j
        self.mid = self.k[0]
        t = self.k[1] / self.k[1].norm(dim=1, keepdim=True)
        self.normal = torch.stack([t[:, 1], -t[:, 0]], 1)

    def at(self, a, delta):
        """Positions (relative to alpha = 0 with delta) and |dx/dalpha| at the parameters a (A,)."""
        a = a[None, :, None]
        k0, k1, k2, k3 = (k[:, None] for k in self.k)
        p = a * (k1 + a * (k2 + a * k3))
        d = k1 + a * (2 * k2 + a * 3 * k3)
        return (p if delta else p + k0), d.norm(dim=2)

    def matrix(self, flux):
        """The BEM matrix: potential rows, or (flux: the factor of each row) n . E rows."""
        A = torch.empty((self.n, self.n), dtype=torch.float64, device=self.mid.device)
        rs, zs, w = self.pos[None, :, :, 0], self.pos[None, :, :, 1], self.jac[None]
        step = max(1, 24_000_000 // (16 * self.n))
        for i in range(0, self.n, step):
            m = self.mid[i:i + step]
            A[i:i + step] = (w * self._kernel(m, rs, zs, flux, slice(i, i + step))).sum(2)
        self._diagonal(A, flux)
        return A

    def _kernel(self, m, rs, zs, flux, rows):
        r0, z0 = m[:, 0, None, None], m[:, 1, None, None]
        if flux is None:
            return _ring(r0, z0, rs, zs, 'pot')
        er, ez = _ring(r0, z0, rs, zs, 'field')
        n = self.normal[rows]
        return flux * (n[:, 0, None, None] * er + n[:, 1, None, None] * ez)

    def _diagonal(self, A, flux):
        x, w = np.polynomial.legendre.leggauss(16)
        a, b = [], []
        for lvl in range(53):  # intervals graded geometrically toward the log singularity
            hi = 2.0 ** -lvl
            lo = 0.0 if lvl == 52 else 0.5 * hi
            a.append(0.5 * (hi + lo) + 0.5 * (hi - lo) * x)
            b.append(0.5 * (hi - lo) * w)
        a, b = np.concatenate(a), np.concatenate(b)
        a, b = (torch.as_tensor(np.concatenate([s * u, u2]), device=A.device) for s, u, u2 in ((-1, a, a), (1, b, b)))
        for i in range(0, self.n, 4096):
            s = slice(i, min(self.n, i + 4096))
            e = _Elements.__new__(_Elements)
            e.k = [k[s] for k in self.k]
            d, j = e.at(a, True)
            r0 = self.mid[s][:, 0, None]
            dr, dz = d[..., 0], d[..., 1]
            rho2, rs = dr * dr + dz * dz, r0 + dr
            D = rho2 + 4 * r0 * rs
            K, E = _elliptic(rho2 / D)
            q = rs / (math.pi * torch.sqrt(D))
            if flux is None:
                v = (b * j * q * K).sum(1)
            else:
                er = q * (rho2 * (K - E) - 2.0 * r0 * dr * E) / (2.0 * r0 * rho2)
                ez = -q * dz * E / rho2
                n = self.normal[s]
                v = (b * j * flux * (n[:, 0, None] * er + n[:, 1, None] * ez)).sum(1) - 1.0
            idx = torch.arange(s.start, s.stop, device=A.device)
            A[idx, idx] = v

    def solve(self, F, flux=None):
        """Charges (nrhs, N) for the right-hand sides F (nrhs, N)."""
        return torch.linalg.solve(self.matrix(flux), torch.as_tensor(F, device=self.mid.device).T).T.contiguous()


class _Sources:
    """Rings (r, z, w) of electric charges, magnetic charges and coils, and their fields."""

    def __init__(self, elec=None, mag=None, coil=None):
        self.elec, self.mag, self.coil = elec, mag, coil

    @staticmethod
    def _sum(p, rings, fn):
        r, z, w = rings
        r0 = torch.clamp(torch.hypot(p[:, 0], p[:, 1]), min=1e-12)[:, None]
        out = torch.empty((2, len(p)), dtype=torch.float64, device=p.device)
        step = max(1, 24_000_000 // len(r))
        for i in range(0, len(p), step):
            fr, fz = fn(r0[i:i + step], p[i:i + step, 2:3], r[None], z[None])
            out[0, i:i + step], out[1, i:i + step] = fr @ w, fz @ w
        c = out[0] / r0[:, 0]
        return torch.stack([p[:, 0] * c, p[:, 1] * c, out[1]], 1)

    def E(self, p):
        return self._sum(p, self.elec, lambda *a: _ring(*a, 'field')) if self.elec else torch.zeros_like(p)

    def H(self, p):
        h = self._sum(p, self.mag, lambda *a: _ring(*a, 'field')) if self.mag else torch.zeros_like(p)
        return h + self._sum(p, self.coil, _coil) if self.coil else h


def _rings(el, q):
    return (el.pos[..., 0].reshape(-1), el.pos[..., 1].reshape(-1), (q[:, None] * el.jac).reshape(-1))


def _coil_rings(coils):
    I, jac, pos = coils
    return tuple(torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device=_dev())
                 for a in (pos[..., 0], pos[..., 2], I[:, None] * jac))


RK_B = [[], [2 / 9], [1 / 12, 1 / 4], [69 / 128, -243 / 128, 135 / 64], [-17 / 12, 27 / 4, -27 / 5, 16 / 15],
        [65 / 432, -5 / 16, 13 / 16, 4 / 27, 5 / 144]]
RK_CH = [47 / 450, 0, 12 / 25, 32 / 225, 1 / 30, 6 / 25]
RK_CT = [-1 / 150, 0, 3 / 100, -16 / 75, -1 / 20, 6 / 25]


def _integrate(field, pos, vel, bounds, atol, plane_z=None):
    """Adaptive RKF45 of all electrons in step: final states (n, 7) and crossings of z = plane_z (n, 7)."""
    from traceon_b200.tracing import e as charge, m_e
    dev, qm = _dev(), -charge / m_e
    y = torch.as_tensor(np.concatenate([pos, vel], 1), device=dev)
    lo, hi = (torch.as_tensor(np.ascontiguousarray(np.asarray(bounds)[:, i]), device=dev) for i in (0, 1))
    n = len(y)
    t = torch.zeros(n, dtype=torch.float64, device=dev)
    hmax = 0.01 / y[:, 3:].norm(dim=1)
    h = hmax.clone()
    plane = torch.full((n, 7), float('nan'), dtype=torch.float64, device=dev)
    live = torch.arange(n, device=dev)
    for _ in range(5000):
        live = live[((lo <= y[live, :3]) & (y[live, :3] <= hi)).all(1)]
        if not len(live):
            break
        Y, H = y[live], h[live, None]
        k = []
        for s in range(6):
            ys = Y + sum((b * kk for b, kk in zip(RK_B[s], k)), torch.zeros_like(Y))
            E, B = field(ys[:, :3])
            a = qm * (E + MU0 * torch.linalg.cross(ys[:, 3:], B))
            k.append(H * torch.cat([ys[:, 3:], a], 1))
        e = sum(c * kk for c, kk in zip(RK_CT, k)).abs()
        err = e[:, :3].max(1).values + h[live] * e[:, 3:].max(1).values
        ok = err <= atol
        new = Y + sum(c * kk for c, kk in zip(RK_CH, k))
        if plane_z is not None:
            cross = ok & ((Y[:, 2] - plane_z > 0) != (new[:, 2] - plane_z > 0))
            if cross.any():
                plane[live[cross]] = _crossing(H[cross, 0], Y[cross], new[cross], plane_z, t[live[cross]])
        at = live[ok]
        y[at], t[at] = new[ok], t[at] + h[at]
        h[live] = torch.minimum(0.9 * h[live] * (atol / err) ** 0.2, hmax[live])
    return torch.cat([t[:, None], y], 1), plane


def _crossing(h, a, b, zp, t0):
    """Cubic-Hermite crossing of z = zp between the states a and b, a step h apart."""
    def at(u, c):
        u2, u3 = u * u, u * u * u
        return ((2 * u3 - 3 * u2 + 1) * a[:, c] + (u3 - 2 * u2 + u) * h * a[:, 3 + c] + (3 * u2 - 2 * u3) * b[:, c]
                + (u3 - u2) * h * b[:, 3 + c])
    lo, hi = torch.zeros_like(h), torch.ones_like(h)
    above = a[:, 2] > zp
    for _ in range(60):
        u = 0.5 * (lo + hi)
        same = (at(u, 2) > zp) == above
        lo, hi = torch.where(same, u, lo), torch.where(same, hi, u)
    u = 0.5 * (lo + hi)
    out = [t0 + u * h, at(u, 0), at(u, 1), torch.full_like(u, zp)]
    return torch.stack(out + [(1 - u) * a[:, 3 + c] + u * b[:, 3 + c] for c in range(3)], 1)


def _axial_table(rings, z):
    """The axial coefficients (nz - 1, 9, 6) of the rings: quintic Hermite pieces of the derivatives 0..6,
    not-a-knot cubic splines of 7 and 8, highest power first."""
    r, zs, w = rings
    zt = torch.as_tensor(z, device=r.device)
    nz, h = len(z), float(z[1] - z[0])
    d = torch.zeros((nz, 9), dtype=torch.float64, device=r.device)
    step = max(1, 16_000_000 // len(r))
    for i in range(0, nz, step):
        u = zt[i:i + step, None] - zs[None]
        R = torch.hypot(u, r.expand_as(u))
        p0, p1 = torch.ones_like(u), u / R   # derivative n of 1 / R: (-1)^n n! P_n(u / R) / R^(n + 1)
        f = 0.5 * w * r / R
        for n in range(9):
            d[i:i + step, n] = (f * p0).sum(1)
            f = f * (-(n + 1.0)) / R
            p0, p1 = p1, ((2 * n + 3) * (u / R) * p1 - (n + 1) * p0) / (n + 2)
    c = torch.zeros((nz - 1, 9, 6), dtype=torch.float64, device=r.device)
    for i in range(7):
        c0, c1, c2 = d[:-1, i], d[:-1, i + 1], 0.5 * d[:-1, i + 2]
        D0 = d[1:, i] - (c0 + h * (c1 + h * c2))
        D1 = (d[1:, i + 1] - (c1 + 2 * h * c2)) * h
        D2 = (d[1:, i + 2] - 2 * c2) * h * h
        c[:, i] = torch.stack([(6 * D0 - 3 * D1 + 0.5 * D2) / h ** 5, (-15 * D0 + 7 * D1 - D2) / h ** 4,
                               (10 * D0 - 4 * D1 + 0.5 * D2) / h ** 3, c2, c1, c0], 1)
    T = torch.zeros((nz, nz), dtype=torch.float64, device=r.device)
    k = torch.arange(1, nz - 1, device=r.device)
    T[k, k - 1], T[k, k], T[k, k + 1] = 1.0, 4.0, 1.0
    T[0, 0], T[0, 2], T[-1, -1], T[-1, -3] = 1.0, -1.0, 1.0, -1.0
    m = (d[1:, 7:] - d[:-1, 7:]) / h
    rhs = torch.cat([2 * (m[:1] - m[1:2]), 3 * (m[:-1] + m[1:]), 2 * (m[-1:] - m[-2:-1])])
    s = torch.linalg.solve(T, rhs)
    for q in range(2):
        s0, s1, mq = s[:-1, q], s[1:, q], m[:, q]
        c[:, 7 + q, 2:] = torch.stack([(s0 + s1 - 2 * mq) / h ** 2, (3 * mq - 2 * s0 - s1) / h, s0, d[:-1, 7 + q]], 1)
    return c


def _axial_field(c, z, p):
    """The field of the radial series of an axial table at the points p."""
    zt = torch.as_tensor(z, device=p.device)
    inside = (zt[0] <= p[:, 2]) & (p[:, 2] <= zt[-1])
    idx = ((p[:, 2] - zt[0]) / (zt[1] - zt[0])).long().clamp(0, len(z) - 2)
    x = (p[:, 2] - zt[idx])[:, None]
    d = torch.zeros((len(p), 9), dtype=torch.float64, device=p.device)
    for i in range(6):
        d = d * x + c[idx, :, i]
    r2 = p[:, 0] ** 2 + p[:, 1] ** 2
    fr = 0.5 * (d[:, 2] - r2 / 8 * d[:, 4] + r2 ** 2 / 192 * d[:, 6] - r2 ** 3 / 9216 * d[:, 8])
    fz = -d[:, 1] + r2 / 4 * d[:, 3] - r2 ** 2 / 64 * d[:, 5] + r2 ** 3 / 2304 * d[:, 7]
    return torch.where(inside[:, None], torch.stack([p[:, 0] * fr, p[:, 1] * fr, fz], 1), torch.zeros_like(p))


# ---------------------------------------------------------------- inputs
def _lens(n_el, seed):
    """The einzel lens, its voltages, and its charges."""
    from traceon_b200 import geometry as G
    geo = G.einzel_lens(n_el)
    el = _Elements(geo.vertices)
    volts = G.einzel_lens_voltages(seed)
    return geo, el, el.solve(geo.voltages_to_values(volts)[None])[0]


def _pole(n_el, seed):
    """The pole piece of the combined lens with its coils, and its magnetic charges."""
    from traceon_b200 import geometry as G
    lens = G.combined_lens(seed, n_elec=60, n_mag=n_el)
    geo = lens.geometry
    pole = geo.vertices[geo.electrode_index == 3]
    el = _Elements(pole)
    coils = lens.coil_sources()
    f = _flux(1000.0)
    return lens, el, el.solve(_pole_rhs(el, coils, f)[None], f)[0], coils


def _flux(mu):
    return 2.0 * (mu - 1) / (1 + mu)


def _pole_rhs(el, coils, f):
    p = torch.stack([el.mid[:, 0], torch.zeros_like(el.mid[:, 0]), el.mid[:, 1]], 1)
    h = _Sources(coil=_coil_rings(coils)).H(p)
    return -f * (h[:, 0] * el.normal[:, 0] + h[:, 2] * el.normal[:, 1])


def _points(n, seed, r_max):
    rng = np.random.default_rng(seed)
    r, phi = rng.uniform(0.01 * MM, r_max, n), rng.uniform(0, 2 * np.pi, n)
    return np.stack([r * np.cos(phi), r * np.sin(phi), rng.uniform(-8 * MM, 8 * MM, n)], 1)


def _point_charges(el, q):
    from traceon_b200.field import EffectivePointCharges
    return EffectivePointCharges(q.cpu().numpy(), el.jac.cpu().numpy(), el.pos.cpu().numpy())


def _pole_field(el, q, coils):
    from traceon_b200.field import EffectivePointCharges, FieldRadialBEM
    return FieldRadialBEM(magnetostatic_point_charges=_point_charges(el, q),
                          current_point_charges=EffectivePointCharges(*coils))


def _stacks(case, seed):
    """Lens stacks of uneven size with voltages well below the beam's, and their beams."""
    from traceon_b200 import geometry as G
    out = []
    for g in range(case['lenses']):
        geo, _ = G.random_lens(g, n_range=(300, case['n_max']))
        v = np.random.default_rng([seed, g]).uniform(-500.0, 500.0, len(geo.names))
        z0, z1 = geo.segments[:, [1, 3]].min(), geo.segments[:, [1, 3]].max()
        h = 0.9 * geo.segments[1::3, 2].min()
        pos, vel = G.electron_beam(case['electrons'], seed + g, z0=z0 - 0.5 * MM, r_max=0.05 * MM, angle_max=2e-3,
                                   energy_spread=0.05)
        out.append((geo, geo.voltages_to_values(v), v, pos, vel,
                    np.array([[-h, h], [-h, h], [z0 - 1 * MM, z1 + 1 * MM]])))
    return out


def _single(case, seed):
    from traceon_b200 import geometry as G
    geo, el, q = _lens(case['n_el'] // 2, seed)
    _, pel, pq, coils = _pole(case['n_el'] - case['n_el'] // 2, seed)
    pos, vel = G.combined_beam(1, seed)
    return el, q, pel, pq, coils, pos, vel


def _unit_charges(n_el):
    from traceon_b200 import geometry as G
    geo = G.einzel_lens(n_el)
    el = _Elements(geo.vertices)
    return geo, el, el.solve(geo.unit_rhs())


def _excitation(geo, values):
    from traceon_b200.excitation import Excitation, Mesh
    exc = Excitation(Mesh.from_geometry(geo))
    exc.add_voltage(**{n: float(v) for n, v in zip(geo.names, values)})
    return exc


def prepare(case, seed):
    from traceon_b200 import geometry as G
    from traceon_b200.field import FieldRadialAxial, FieldRadialBEM
    kind, s = case['kind'], {'case': case}
    if kind in ('point', 'axial', 'trace_axial', 'trace_bem') or (kind == 'map' and not case['magnetic']):
        geo, el, q = _lens(case['n_el'], seed)
        s['field'] = FieldRadialBEM(electrostatic_point_charges=_point_charges(el, q))
    if kind == 'point':
        s['point'] = _points(1, seed, 0.9 * MM)[0]
    elif kind == 'map':
        s['points'] = _points(case['points'], seed, (2.3 if case['magnetic'] else 0.9) * MM)
        if case['magnetic']:
            s['field'] = _pole_field(*_pole(case['n_el'], seed)[1:])
    elif kind == 'solve':
        rng = np.random.default_rng(seed)
        geo = G.einzel_lens(case['n_el'])
        s['excitation'] = _excitation(geo, [1.0, 1.0, 1.0])
        s['F'] = rng.uniform(-3000, 3000, (case['nrhs'], 3)) @ geo.unit_rhs()
    elif kind == 'solve_magnetic':
        from traceon_b200.excitation import Excitation, Mesh
        from traceon_b200.field import EffectivePointCharges
        lens = G.combined_lens(seed, n_elec=60, n_mag=case['n_el'])
        s['excitation'] = Excitation(Mesh.from_geometry(lens.geometry))
        s['excitation'].add_magnetizable(pole=1000.0)
        s['coils'] = EffectivePointCharges(*lens.coil_sources())
    elif kind == 'sweep':
        from traceon_b200.batch import BatchPipeline
        st = _stacks(case, seed)
        s['pipeline'] = BatchPipeline([_excitation(x[0], x[2]) for x in st], [x[3] for x in st], [x[4] for x in st],
                                      [x[5] for x in st], atol=1e-9)
        s['pipeline'].capture()
    elif kind in ('trace_axial', 'trace_bem'):
        s['beam'] = G.surrogate_beam(case['electrons'], seed, r_max=0.35 * MM)
        f = s['field']
        if kind == 'trace_axial':
            f = FieldRadialAxial(f, -11.5 * MM, 11.5 * MM, case['nz'])
        s['tracer'] = f.get_tracer(G.LENS_BOUNDS)
    elif kind == 'trace_single':
        el, q, pel, pq, coils, pos, vel = _single(case, seed)
        f = FieldRadialBEM(electrostatic_point_charges=_point_charges(el, q)) + _pole_field(pel, pq, coils)
        s['tracer'], s['start'] = f.get_tracer(G.LENS_BOUNDS), (pos, vel)
    elif kind == 'trace_surrogate':
        from traceon_b200 import surrogate as S
        geo, el, q = _unit_charges(case['n_el'])
        fields = [FieldRadialBEM(electrostatic_point_charges=_point_charges(el, x)) for x in q]
        z, _, tabs = S.axial_tables(fields, -11.5 * MM, 11.5 * MM, 4601)
        scale = np.tile([1e-3, 5.0, 5.0], 11)[:32]  # per volt: V, V/m, V/m at r_max
        model = S.SurrogateModel(3, 0.75 * MM, -11.5 * MM, 11.5 * MM, scale, seed=seed)
        fs = S.FieldSurrogate(model, fields, z, tabs, G.einzel_lens_voltages(seed), geo.segments)
        s['session'] = fs.trace_session(case['electrons'], G.LENS_BOUNDS, G.LENS_EXIT_Z, atol=1e-10)
        s['beam'] = G.surrogate_beam(case['electrons'], seed, r_max=0.35 * MM)
    elif kind == 'train':
        from traceon_b200 import surrogate as S
        params, X, T, w, m, v = _train_inputs(case, seed)
        s['mlp'] = S.MLP(params=params)
        s['mlp'].m.copy_(m)
        s['mlp'].v.copy_(v)
        s['mlp'].step_count = 1000
        s['X'], s['T'], s['w'] = X, T, w
    return s


def _train_inputs(case, seed):
    """A network and its optimiser state in mid-training, and one batch of weighted samples."""
    from traceon_b200 import surrogate as S
    rng = np.random.default_rng(seed)
    p = np.zeros(S.NPARAM, dtype=np.float32)
    for W, b, fan_in, _ in S.LAYERS:
        o, n = S.OFF[W]
        p[o:o + n] = rng.uniform(-1, 1, n) * math.sqrt(6.0 / fan_in)
        o, n = S.OFF[b]
        p[o:o + n] = rng.uniform(-0.1, 0.1, n)
    M = case['batch']
    rho2, zeta = rng.uniform(0.02, 1, M), rng.uniform(-1, 1, M)
    X = [rho2, zeta, rho2 * zeta, zeta ** 2, rho2 ** 2, rho2 * zeta ** 2]
    for k in range(1, 6):
        X += [np.sin(k * np.pi * zeta), np.cos(k * np.pi * zeta)]
    f = (lambda a, t: torch.as_tensor(np.asarray(a), device=_dev()).to(t).contiguous())
    T = np.sin(3 * zeta)[:, None] * rng.uniform(0.5, 1.5, 3 * case['n_src']) + 0.1 * rng.standard_normal((M, 3 * case['n_src']))
    return (p, f(np.stack(X, 1), torch.bfloat16), f(T, torch.float32), f(rng.uniform(0.2, 3, M), torch.float32),
            f(rng.standard_normal(S.NPARAM) * 1e-4, torch.float32), f(rng.uniform(0.5, 2, S.NPARAM) * 1e-6, torch.float32))


# ---------------------------------------------------------------- one pass
def run(s):
    case = s['case']
    kind = case['kind']
    if kind == 'point':
        return s['field'].electrostatic_field_at_point(s['point'])
    if kind == 'map':
        if case['magnetic']:
            return s['field'].magnetostatic_field_at_points(s['points'])
        return s['field'].electrostatic_field_at_points(s['points'])
    if kind == 'solve':
        from traceon_b200.solver import ElectrostaticSolverRadial
        fields = ElectrostaticSolverRadial(s['excitation']).solve_matrix(s['F'])
        return [f.electrostatic_point_charges.charges for f in fields]
    if kind == 'solve_magnetic':
        from traceon_b200.solver import MagnetostaticSolverRadial
        f = MagnetostaticSolverRadial(s['excitation'], s['coils']).solve_matrix()[0]
        return f.magnetostatic_point_charges.charges
    if kind == 'sweep':
        p = s['pipeline']
        p.replay()
        res = p.results()
        return {'charges': p.batch.charges, 'final': [r[0] for r in res], 'status': [r[1] for r in res],
                'counters': [r[2] for r in res]}
    if kind == 'axial':
        from traceon_b200.field import FieldRadialAxial
        return FieldRadialAxial(s['field'], -11.5 * MM, 11.5 * MM, case['nz']).electrostatic_coeffs
    if kind in ('trace_axial', 'trace_bem'):
        plane, final, status, counters = s['tracer'].trace_endpoints(*s['beam'], 9.5 * MM, atol=10.0 ** case['log_atol'])
        return {'plane': plane, 'final': final, 'status': status, 'counters': counters}
    if kind == 'trace_single':
        plane, final, status, counters = s['tracer'].trace_endpoints(*s['start'], 9.5 * MM, atol=1e-9)
        return {'plane': plane, 'final': final, 'status': status, 'counters': counters}
    if kind == 'trace_surrogate':
        plane, final, status, counters = s['session'].run(*s['beam'])
        return {'plane': plane, 'final': final, 'status': status, 'counters': counters}
    mlp = s['mlp']
    loss = mlp.loss_and_grad(s['X'], s['T'], 3 * case['n_src'], s['w'])
    mlp.adam(1e-3)
    return {'loss': loss, 'grad': mlp.g, 'params': mlp.p}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case['kind']
    n = case.get('n_el', 0)
    rings = 16 * n * 24
    if kind == 'point':
        return {'bytes': rings + 48, 'flops': RING_FLOPS * n}
    if kind == 'map':
        return {'bytes': rings + 48 * case['points'], 'flops': RING_FLOPS * n * case['points']}
    if kind in ('solve', 'solve_magnetic'):
        nrhs = case.get('nrhs', 1)
        return {'bytes': 96 * n + 16 * nrhs * n, 'flops': 2 / 3 * n ** 3 + 2 * nrhs * n * n + 50 * n * n}
    if kind == 'sweep':
        m = 0.5 * (300 + case['n_max'])
        e = case['lenses'] * case['electrons']
        return {'bytes': case['lenses'] * 112 * m + 108 * e,
                'flops': case['lenses'] * (2 / 3 * m ** 3 + 50 * m * m) + e * 6 * ATTEMPTS * RING_FLOPS * m}
    if kind == 'axial':
        return {'bytes': rings + 432 * case['nz'], 'flops': 54 * n * case['nz']}
    if kind == 'trace_axial':
        return {'bytes': 432 * case['nz'] + 188 * case['electrons'], 'flops': 400 * ATTEMPTS * 6 * case['electrons']}
    if kind == 'trace_bem':
        return {'bytes': rings + 188 * case['electrons'], 'flops': RING_FLOPS * n * 6 * ATTEMPTS * case['electrons']}
    if kind == 'trace_single':
        return {'bytes': rings + 56 * ATTEMPTS, 'flops': RING_FLOPS * n * 6 * ATTEMPTS}
    if kind == 'trace_surrogate':
        return {'bytes': 188 * case['electrons'] + 432 * 4600, 'flops': EVAL_FLOPS * 6 * ATTEMPTS * case['electrons']}
    return {'bytes': case['batch'] * (36 + 12 * case['n_src']) + 51360 * 32, 'flops': 3 * EVAL_FLOPS * case['batch']}


# ---------------------------------------------------------------- the same in plain 64-bit arithmetic
def exact(case, seed):
    """What run() returns; None where plain arithmetic takes too long (the largest maps and beams) or has no
    such value (integers; the surrogate, whose network is evaluated in 16 bits by design)."""
    kind = case['kind']
    none = {'plane': None, 'final': None, 'status': None, 'counters': None}
    if kind == 'point':
        _, el, q = _lens(case['n_el'], seed)
        p = torch.as_tensor(_points(1, seed, 0.9 * MM), device=_dev())
        return _Sources(elec=_rings(el, q)).E(p)[0].cpu().numpy()
    if kind == 'map':
        if case['n_el'] * case['points'] > 200_000_000:
            return None
        p = torch.as_tensor(_points(case['points'], seed, (2.3 if case['magnetic'] else 0.9) * MM), device=_dev())
        if case['magnetic']:
            _, el, q, coils = _pole(case['n_el'], seed)
            return _Sources(mag=_rings(el, q), coil=_coil_rings(coils)).H(p).cpu().numpy()
        _, el, q = _lens(case['n_el'], seed)
        return _Sources(elec=_rings(el, q)).E(p).cpu().numpy()
    if kind == 'solve':
        from traceon_b200 import geometry as G
        geo = G.einzel_lens(case['n_el'])
        F = np.random.default_rng(seed).uniform(-3000, 3000, (case['nrhs'], 3)) @ geo.unit_rhs()
        return list(_Elements(geo.vertices).solve(F).cpu().numpy())
    if kind == 'solve_magnetic':
        return _pole(case['n_el'], seed)[2].cpu().numpy()
    if kind == 'sweep':
        charges, final = [], []
        for geo, values, _, pos, vel, bounds in _stacks(case, seed):
            el = _Elements(geo.vertices)
            charges.append(el.solve(values[None])[0])
            src = _Sources(elec=_rings(el, charges[-1]))
            final.append(_integrate(lambda p: (src.E(p), torch.zeros_like(p)), pos, vel, bounds, 1e-9)[0].cpu().numpy())
        return {'charges': charges, 'final': final, 'status': [None] * len(final), 'counters': [None] * len(final)}
    if kind == 'axial':
        _, el, q = _lens(case['n_el'], seed)
        return _axial_table(_rings(el, q), np.linspace(-11.5 * MM, 11.5 * MM, case['nz'])).cpu().numpy()
    if kind in ('trace_axial', 'trace_bem'):
        from traceon_b200 import geometry as G
        if kind == 'trace_bem' and case['n_el'] * case['electrons'] > 1_000_000:
            return None
        _, el, q = _lens(case['n_el'], seed)
        src = _Sources(elec=_rings(el, q))
        z = np.linspace(-11.5 * MM, 11.5 * MM, case.get('nz', 2))
        c = _axial_table(src.elec, z) if kind == 'trace_axial' else None
        pos, vel = G.surrogate_beam(case['electrons'], seed, r_max=0.35 * MM)
        final, plane = _integrate(lambda p: (src.E(p) if c is None else _axial_field(c, z, p), torch.zeros_like(p)),
                                     pos, vel, G.LENS_BOUNDS, 10.0 ** case['log_atol'], 9.5 * MM)
        return {**none, 'plane': plane.cpu().numpy(), 'final': final.cpu().numpy()}
    if kind == 'trace_single':
        from traceon_b200 import geometry as G
        el, q, pel, pq, coils, pos, vel = _single(case, seed)
        src = _Sources(_rings(el, q), _rings(pel, pq), _coil_rings(coils))
        final, plane = _integrate(lambda p: (src.E(p), src.H(p)), pos, vel, G.LENS_BOUNDS, 1e-9, 9.5 * MM)
        return {**none, 'plane': plane.cpu().numpy(), 'final': final.cpu().numpy()}
    if kind == 'trace_surrogate':
        return None
    return _train_exact(case, seed)


def _train_exact(case, seed):
    from traceon_b200 import surrogate as S
    params, X, T, w, m, v = (a.double() if isinstance(a, torch.Tensor) else a for a in _train_inputs(case, seed))
    p = torch.as_tensor(params, dtype=torch.float64, device=X.device).requires_grad_()
    y = X
    for i, (W, b, fin, fout) in enumerate(S.LAYERS):
        y = y @ p[S.OFF[W][0]:S.OFF[W][0] + fin * fout].reshape(fout, fin).T + p[S.OFF[b][0]:S.OFF[b][0] + fout]
        if i < 4:
            y = torch.nn.functional.silu(y)
    loss = (w[:, None] * (y[:, :T.shape[1]] - T) ** 2).sum() / T.numel()
    g, = torch.autograd.grad(loss, p)
    m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
    step = 1e-3 * (m / (1 - 0.9 ** 1001)) / (torch.sqrt(v / (1 - 0.999 ** 1001)) + 1e-8)
    return {'loss': loss.detach(), 'grad': g, 'params': (p - step).detach()}
