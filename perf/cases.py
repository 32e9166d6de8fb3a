"""The work that users of this framework have it do, as cases that can be timed.

A case is one configuration (flavors, cells, directions per cell, stencil
order, precision) and one way of driving it through the Python binding:

  evolve   the run loop between two outputs: `steps` device-resident RK4 steps
           (Context.evolve), then the particles come back to the host, and,
           where `mesh` is set, the deposited fields too (a plotfile's
           content).  A pass goes on from the state the last one left, as the
           next output interval of a run does.
  loop     a host that keeps its own integrator loop: compute_dt and step for
           each step, then the derivatives, the fields and the particles.
  adjoint  a gradient: load, recorded forward run, objective, backward sweep.

Particles are the ones of the sample problems: one set of directions at the
centre of every cell, 50 MeV, electron flavor with a seeded off-diagonal
perturbation of 1e-6, nu_e isotropic and nubar_e with a flux factor.
"""
import math

import numpy as np
import torch
import torch.utils.checkpoint

from emu_b200 import api

EV, C, HBAR, MP = 1.60218e-12, 2.99792458e10, 1.05457266e-27, 1.6726219e-24
HBARC = HBAR * C
GF = 1.1663787e-5 / (1e9 * 1e9 * EV * EV) * HBARC * HBARC * HBARC
PUPT = 50e6 * EV
DEG = math.pi / 180.0
B = (1.0 / 6.0, 1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0)


def _case(name, how, nf, nx, ny, nz, dirs, steps, precision="fp64", order=2, mesh=False, interval=0, msw=False):
    return {"name": name, "how": how, "nf": nf, "nx": nx, "ny": ny, "nz": nz, "dirs": dirs, "steps": steps,
            "precision": precision, "order": order, "mesh": mesh, "interval": interval, "msw": msw}


def listed():
    return [
        # the smallest run: vacuum and matter oscillation of two particles in
        # one cell (the MSW test), 50 steps: launch latency
        _case("msw_one_cell", "evolve", 2, 1, 1, 1, 2, 50, msw=True, mesh=True),
        # the k != 0 instability test: 50 cells of two beams
        _case("beams_1d", "evolve", 2, 1, 1, 50, 2, 100, mesh=True),
        # fast-flavor instability in 1D, two flavors (128 cells, 80 directions)
        _case("fast_flavor_1d", "evolve", 2, 1, 1, 128, 80, 50, mesh=True),
        # the fiducial 1D run, three flavors (256 cells, 92 directions)
        _case("fiducial_1d", "evolve", 3, 1, 1, 256, 92, 30, mesh=True),
        # the large 1D run in mixed precision (1024 cells, 378 directions)
        _case("wide_1d_mixed", "evolve", 3, 1, 1, 1024, 378, 30, "mixed"),
        # a host that drives single steps itself, linear (CIC) shape factors,
        # an odd number of cells
        _case("host_loop_cic", "loop", 2, 1, 1, 201, 50, 10, order=1, mesh=True),
        # a two-dimensional run, ragged extents
        _case("plane_2d", "evolve", 3, 1, 90, 77, 60, 5, mesh=True),
        # 3D, double precision (32^3 cells, 96 directions)
        _case("box_3d", "evolve", 3, 32, 32, 32, 96, 5, mesh=True),
        # 3D, two flavors, mixed precision, odd extents
        _case("box_3d_two_flavors_mixed", "evolve", 2, 27, 25, 29, 50, 10, "mixed"),
        # the largest run: 3D, mixed precision (64^3 cells, 96 directions)
        _case("box_3d_mixed", "evolve", 3, 64, 64, 64, 96, 10, "mixed"),
        # gradient of the 1D fast-flavor run, checkpoints every 25 steps
        _case("adjoint_1d", "adjoint", 2, 1, 1, 128, 80, 50, interval=25),
        # gradient of a 3D three-flavor run
        _case("adjoint_3d", "adjoint", 3, 16, 16, 16, 48, 10, interval=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: 1D to 3D, any extents, both precisions."""
    how = rng.choice(["evolve"] * 6 + ["loop", "adjoint"])
    dims = rng.choice([1, 1, 2, 3, 3])
    nf = rng.choice([2, 3])
    precision = rng.choice(["fp64", "mixed"]) if how == "evolve" else "fp64"
    order = 2 if how != "loop" else rng.choice([1, 2])
    dirs = rng.randint(20, 130) if dims > 1 else _log_int(rng, 2, 378)
    if dims == 1:
        n = (1, 1, _log_int(rng, 8, 1024))
    elif dims == 2:
        n = (1, _log_int(rng, 12, 120), _log_int(rng, 12, 120))
    else:
        n = (_log_int(rng, 7, 40), _log_int(rng, 7, 40), _log_int(rng, 7, 40))
    if how == "adjoint":
        n = tuple(min(v, 130 if dims == 1 else 40 if dims == 2 else 15) for v in n)
        dirs = min(dirs, 60)
    steps = {"evolve": rng.randint(20, 50) if dims == 1 else rng.randint(5, 12), "loop": rng.randint(4, 12),
             "adjoint": rng.randint(20, 50) if dims == 1 else rng.randint(5, 10)}[how]
    c = _case("", how, nf, n[0], n[1], n[2], dirs, steps, precision, order,
              mesh=how != "adjoint" and precision == "fp64", interval=rng.choice([5, 10, 25]) if how == "adjoint" else 0)
    del c["name"]
    return c


# ---- inputs -------------------------------------------------------------------
def _params(case, seed):
    cells = (case["nx"], case["ny"], case["nz"])
    dx = 1.0 if case["msw"] else 0.5
    p = api.default_params(nflavors=case["nf"], shape_order=case["order"], ncell=cells, simulation_type=4,
                           Lx=dx * cells[0], Ly=dx * cells[1], Lz=dx * cells[2], cfl_factor=0.5,
                           flavor_cfl_factor=0.5, maxError=1e-6, Ye_in=1.0, seed=seed)
    p.precision = api.PREC_MIXED if case["precision"] == "mixed" else api.PREC_FP64
    g = EV / C ** 2
    if case["nf"] == 2:
        p.mass1, p.mass2, p.mass3 = -0.008596511 * g, 0.0, 0.0
    else:
        p.mass1, p.mass2, p.mass3 = 0.0, 0.0, 0.049487372 * g
    p.theta12 = (33.82 if case["msw"] else 1e-6) * DEG
    p.theta13, p.theta23, p.deltaCP = 48.3 * DEG, 8.61 * DEG, 222.0 * DEG
    if case["msw"]:
        p.rho_in, p.cfl_factor, p.flavor_cfl_factor = 1346160134.709288, 0.5, 0.1
    return p


def _re(nf, i, j):
    return i * (2 * nf - i) + (0 if i == j else 2 * (j - i) - 1)


def _columns(nf):
    """record columns: (f, fbar) reals, (N, Nbar), (L, Lbar)"""
    nh = nf * nf
    return (list(range(13, 13 + nh)) + list(range(15 + nh, 15 + 2 * nh)), [11, 13 + nh], [12, 14 + nh])


def _records(case, seed):
    """particle records [n, nreal], FP64, on the GPU (the CPU without one)"""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    nf, nd = case["nf"], case["dirs"]
    cells = (case["nx"], case["ny"], case["nz"])
    nc, nh = cells[0] * cells[1] * cells[2], nf * nf
    k = torch.arange(nd, dtype=torch.float64, device=dev) + 0.5
    if nd == 2:
        u = torch.tensor([[0.0, 0.0, 1.0], [0.0, 0.0, -1.0]], dtype=torch.float64, device=dev)
    else:
        mu, phi = 1.0 - 2.0 * k / nd, math.pi * (1.0 + math.sqrt(5.0)) * k
        s = torch.sqrt(1.0 - mu * mu)
        u = torch.stack([s * torch.cos(phi), s * torch.sin(phi), mu], 1)
    dx = 1.0 if case["msw"] else 0.5
    r = torch.zeros((nc, nd, 3 + 8 + 2 * (2 + nh)), dtype=torch.float64, device=dev)
    c = torch.arange(nc, device=dev)
    for d, i in enumerate((c // (cells[1] * cells[2]), (c // cells[2]) % cells[1], c % cells[2])):
        r[:, :, d] = ((i.double() + 0.5) * dx)[:, None]
        r[:, :, 4 + d] = r[:, :, d]
        r[:, :, 7 + d] = u[None, :, d] * PUPT
    r[:, :, 10] = PUPT
    fcols, ncols, lcols = _columns(nf)
    gen = torch.Generator(device=dev)
    gen.manual_seed(1000003 * seed + 17)
    for sp in range(2):
        f0 = fcols[sp * nh]
        r[:, :, f0] = 1.0
        amp = 1e-2 if case["msw"] else 1e-6
        for j in range(1, nf):
            for q in (0, 1):
                x = torch.rand((nc, nd), generator=gen, dtype=torch.float64, device=dev)
                r[:, :, f0 + _re(nf, 0, j) + q] = amp * (2.0 * x - 1.0)
        n = 4.89e32 * dx ** 3 / nd
        if case["msw"]:
            r[:, :, ncols[sp]] = 1.0
        else:
            r[:, :, ncols[sp]] = n * (1.0 + (u[None, :, 2] if sp else 0.0))
        f = r[:, :, f0:f0 + nh]
        off = sum(f[:, :, _re(nf, i, j) + q] ** 2 for i in range(nf) for j in range(i + 1, nf) for q in (0, 1))
        r[:, :, lcols[sp]] = torch.sqrt(off + sum(t * t for t in _cartan(f, nf)))
    return r.reshape(nc * nd, -1)


def _cartan(f, nf):
    for m in range(1, nf):
        cl = math.sqrt(2.0 / (m * (m + 1.0))) / 2.0
        yield cl * sum(f[..., _re(nf, i, i)] for i in range(m)) - (cl * m) * f[..., _re(nf, m, m)]


class _State:
    """a context with its particles loaded, and the host buffer that they came
    from and go back to"""

    def __init__(self, case, seed):
        self.case = dict(case)
        self.nf = case["nf"]
        r = _records(case, seed)
        self.n = r.shape[0]
        self.host = torch.empty(r.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
        self.host.copy_(r)
        del r
        if torch.cuda.is_available():
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
        self.ctx = api.Context(_params(case, seed))
        self.ctx.load_particles_ptr(self.host.data_ptr(), self.n)
        self.time = 0.0
        self.out = torch.empty_like(self.host) if case["how"] == "loop" else self.host


def prepare(case, seed):
    return _State(case, seed)


def _particles(records, nf):
    f, _, _ = _columns(nf)
    return {"position": records[:, 0:3], "time": records[:, 3], "momentum": records[:, 7:11],
            "flavor": records[:, f[0]:f[0] + nf * nf], "flavorbar": records[:, f[nf * nf]:f[nf * nf] + nf * nf]}


def _mesh(m, nf, cells):
    return m.reshape(3 + 8 * nf * nf, cells)[3:]


def run(s):
    c = s.case
    nc = c["nx"] * c["ny"] * c["nz"]
    if c["how"] == "adjoint":
        s.ctx.load_particles_ptr(s.host.data_ptr(), s.n)
        dts, _ = s.ctx.adjoint_forward(c["steps"], c["interval"])
        J, lf, lN = s.ctx.adjoint_objective()
        gf, gN = s.ctx.adjoint_backward(lf, lN)
        return {"objective": J, "grad_flavor": gf, "grad_number": gN, "dts": dts}
    if c["how"] == "evolve":
        info = s.ctx.evolve(c["steps"], s.time)
        s.time = info.time
        s.ctx.get_particles_ptr(s.host.data_ptr(), s.n)
        out = _particles(s.host, s.nf)
        if c["mesh"]:
            out["mesh"] = _mesh(s.ctx.get_mesh(), s.nf, nc)
        return out
    for _ in range(c["steps"]):
        dt, _ = s.ctx.compute_dt()
        s.ctx.step(dt)
    rhs = s.ctx.interpolate_rhs()
    f, _, _ = _columns(s.nf)
    s.ctx.get_particles_ptr(s.out.data_ptr(), s.n)
    out = _particles(s.out, s.nf)
    out["rate"] = np.ascontiguousarray(rhs[:, f])
    out["mesh"] = _mesh(s.ctx.get_mesh(), s.nf, nc)
    return out


def work(case):
    nf, nh = case["nf"], case["nf"] ** 2
    n = case["nx"] * case["ny"] * case["nz"] * case["dirs"]
    nreal = 3 + 8 + 2 * (2 + nh)
    width = [1 if m == 1 else case["order"] + 1 for m in (case["nx"], case["ny"], case["nz"])]
    cells = width[0] * width[1] * width[2]
    # a step reads every particle's state (position, time, momentum, weights
    # and lengths, flavor) once and writes position, time and flavor once;
    # the particles come back as records, and with the fields where asked
    step = n * 8.0 * (3 + 1 + 4 + 4 + 2 * nh + 3 + 1 + 2 * nh)
    out = n * 8.0 * nreal + (8.0 * (8 * nh) * n / case["dirs"] if case["mesh"] else 0.0)
    # per stage: a deposit and an interpolation of the nf^2 combinations that
    # the potential holds (number and three fluxes) over the stencil, and two
    # commutators of Hermitian matrices
    stage = n * (2 * 2.0 * cells * 4 * nh + 2 * 8.0 * nf ** 3)
    k = {"evolve": 1.0, "loop": 1.0, "adjoint": 4.0}[case["how"]]
    return {"bytes": k * case["steps"] * step + out, "flops": k * case["steps"] * 4 * stage}


# ---- the same in 64 bits with plain torch ---------------------------------------
class _Exact:
    def __init__(self, case, seed):
        p = _params(case, seed)
        r = _records(case, seed)
        self.nf, self.nh, self.dev = case["nf"], case["nf"] ** 2, r.device
        nf, nh = self.nf, self.nh
        self.cells = [case["nx"], case["ny"], case["nz"]]
        self.L = [p.Lx, p.Ly, p.Lz]
        self.dx = [a / b for a, b in zip(self.L, self.cells)]
        self.vol = self.dx[0] * self.dx[1] * self.dx[2]
        self.order = [case["order"] if m > 1 else 0 for m in self.cells]
        self.p = p
        fcols, ncols, lcols = _columns(nf)
        self.x, self.time = r[:, 0:3].clone(), r[:, 3].clone()
        self.pup = r[:, 7:11].clone()
        self.f, self.N, self.len = r[:, fcols].clone(), r[:, ncols].clone(), r[:, lcols].clone()
        self.v = self.pup[:, :3] / self.pup[:, 3:]
        self.im = torch.zeros(nh, dtype=torch.bool, device=self.dev)
        for i in range(nf):
            for j in range(i + 1, nf):
                self.im[_re(nf, i, j) + 1] = True
        self.sign = torch.where(self.im, -1.0, 1.0).double()
        # vacuum: U diag(m^2) U^+ c^4 / (2 p^t); the sample problems' 2-3
        # rotation is the 1-3 rotation without its phase
        c12, s12 = math.cos(p.theta12), math.sin(p.theta12)
        U = np.eye(nf, dtype=complex)
        U[0, 0] = U[1, 1] = c12
        U[0, 1], U[1, 0] = s12, -s12
        if nf == 3:
            c13, s13 = math.cos(p.theta13), math.sin(p.theta13)
            ph = complex(math.cos(p.deltaCP), -math.sin(p.deltaCP))
            R13 = np.array([[c13, 0, s13 * ph], [0, 1, 0], [-s13 * ph.conjugate(), 0, c13]])
            R23 = np.array([[c13, 0, s13], [0, 1, 0], [-s13, 0, c13]], dtype=complex)
            U = R23 @ R13 @ U
        m2 = np.array([p.mass1 ** 2, p.mass2 ** 2, p.mass3 ** 2][:nf])
        M = U @ np.diag(m2) @ U.conj().T
        c4 = C ** 4
        h = [0.0] * nh
        for i in range(nf):
            h[_re(nf, i, i)] = M[i, i].real
            for j in range(i + 1, nf):
                h[_re(nf, i, j)], h[_re(nf, i, j) + 1] = M[i, j].real, M[i, j].imag
        vac = torch.tensor(h, dtype=torch.float64, device=self.dev)[None, :] * (c4 / (2.0 * self.pup[:, 3:]))
        mat = math.sqrt(2.0) * GF * p.rho_in * p.Ye_in / MP
        self.V0 = [vac.clone(), vac * self.sign]
        self.V0[0][:, 0] += mat
        self.V0[1][:, 0] -= mat
        d = torch.zeros(nh, dtype=torch.float64)
        for i in range(nf):
            d[_re(nf, i, i)] = float(m2[i])
        self.vvac = float(torch.sqrt(sum(t * t for t in _cartan(d, nf)))) * c4 / float(self.pup[:, 3].min())

    def stencil(self, x):
        first, w = [], []
        for d in range(3):
            delta = x[:, d] / self.dx[d]
            near = torch.where(delta - 0.5 < 0.0, delta - 1.0, delta).trunc().long()
            frac = delta - delta.trunc()
            o = torch.where(delta <= 0.0, frac + 0.5, frac - 0.5)
            if self.order[d] == 2:
                first.append(near - 1)
                w.append([0.5 * (0.5 - o) ** 2, 0.75 - o * o, 0.5 * (0.5 + o) ** 2])
            elif self.order[d] == 1:
                first.append(torch.where(o >= 0, near, near - 1))
                w.append([torch.where(o >= 0, 1.0 - o, -o), torch.where(o >= 0, o, 1.0 + o)])
            else:
                first.append(near)
                w.append([torch.ones_like(delta)])
        n = self.cells
        out = []
        for k in range(len(w[2])):
            for j in range(len(w[1])):
                for i in range(len(w[0])):
                    cell = ((torch.remainder(first[2] + k, n[2]) * n[1] + torch.remainder(first[1] + j, n[1])) * n[0]
                            + torch.remainder(first[0] + i, n[0]))
                    out.append((cell, (w[0][i] * w[1][j] * w[2][k])[:, None]))
        return out

    def deposit(self, f, N, st):
        """[cells, 4, 2 nh]: number and fluxes of nu and nubar"""
        nh = self.nh
        fN = torch.cat([f[:, :nh] * N[:, 0:1], f[:, nh:] * N[:, 1:2]], 1)
        val = torch.cat([fN] + [fN * self.v[:, d:d + 1] for d in range(3)], 1)
        m = torch.zeros((self.cells[0] * self.cells[1] * self.cells[2], 8 * nh), dtype=torch.float64, device=self.dev)
        for cell, w in st:
            m = m.index_add(0, cell, val * w) if val.requires_grad else m.index_add_(0, cell, val * w)
        return m

    def _full(self, h):
        nf = self.nf
        rows = []
        for i in range(nf):
            row = []
            for j in range(nf):
                a, b = min(i, j), max(i, j)
                re = h[:, _re(nf, a, b)]
                im = torch.zeros_like(re) if i == j else h[:, _re(nf, a, b) + 1] * (1.0 if i < j else -1.0)
                row.append(torch.complex(re, im))
            rows.append(torch.stack(row, 1))
        return torch.stack(rows, 1)

    def rates(self, f, m, st):
        nf, nh = self.nf, self.nh
        m = m.reshape(-1, 4, 2, nh)
        D = (m[:, :, 0] - self.sign * m[:, :, 1]) * (math.sqrt(2.0) * GF / self.vol)
        G = torch.zeros((f.shape[0], 4, nh), dtype=torch.float64, device=self.dev)
        for cell, w in st:
            G = G + D[cell] * w[:, :, None]
        u = G[:, 0] - sum(self.v[:, d:d + 1] * G[:, 1 + d] for d in range(3))
        out = []
        for sp in range(2):
            H = self._full(self.V0[sp] + (u if sp == 0 else -self.sign * u))
            F = self._full(f[:, sp * nh:(sp + 1) * nh])
            K = (torch.matmul(H, F) - torch.matmul(F, H)) * (-1j / HBAR)
            cols = [None] * nh
            for i in range(nf):
                cols[_re(nf, i, i)] = K[:, i, i].real
                for j in range(i + 1, nf):
                    cols[_re(nf, i, j)], cols[_re(nf, i, j) + 1] = K[:, i, j].real, K[:, i, j].imag
            out += cols
        return torch.stack(out, 1)

    def dt(self, m):
        p, nf, nh = self.p, self.nf, self.nh
        m = m.detach()
        big = max(float(m[:, sp * nh + _re(nf, i, i)].max()) for sp in range(2) for i in range(nf))
        big = max(big, 0.0, self.vol * p.Ye_in * p.rho_in / MP)
        vs = big * (2.0 * nf * math.sqrt(2.0) * GF / self.vol) + self.vvac
        return min(min(self.dx) / C * p.cfl_factor, HBAR / vs * p.flavor_cfl_factor)

    def renormalize(self, f):
        nf, nh, me = self.nf, self.nh, self.p.maxError
        out = []
        for sp in range(2):
            g = list(f[:, sp * nh:(sp + 1) * nh].unbind(1))
            diag = [_re(nf, i, i) for i in range(nf)]
            err = sum(g[d] for d in diag) - 1.0
            for d in diag:
                g[d] = torch.where(err.abs() > me, g[d] - err / nf, g[d])
                g[d] = torch.where(g[d] < -me, torch.zeros_like(g[d]), g[d])
            g = torch.stack(g, 1)
            off = sum(g[:, _re(nf, i, j) + q] ** 2 for i in range(nf) for j in range(i + 1, nf) for q in (0, 1))
            length = torch.sqrt(off + sum(t * t for t in _cartan(g, nf)))
            far = ((length - self.len[:, sp]).abs() > me)[:, None]
            out.append(torch.where(far, g / (length / self.len[:, sp])[:, None], g))
        return torch.cat(out, 1)

    def flavor_step(self, f, N, x, dt):
        """one RK4 step at fixed positions; the last stage's mesh"""
        st = self.stencil(x)
        y, k, new = f, None, f
        for s in range(4):
            if s:
                y = f + (0.5, 0.5, 1.0)[s - 1] * dt * k
            m = self.deposit(y, N, st)
            k = self.rates(y, m, st)
            new = new + dt * B[s] * k
        return self.renormalize(new), m

    def move(self, x, dt):
        x = x + dt * C * self.v
        L = torch.tensor(self.L, dtype=torch.float64, device=self.dev)
        return torch.where(x >= L, x - L, torch.where(x < 0.0, x + L, x))

    def forward(self, steps):
        with torch.no_grad():
            m = self.deposit(self.f, self.N, self.stencil(self.x))
            dts = []
            for _ in range(steps):
                dts.append(self.dt(m))
                self.f, m = self.flavor_step(self.f, self.N, self.x, dts[-1])
                self.x = self.move(self.x, dts[-1])
                self.time = self.time + dts[-1]
        return dts, m


def _out(e):
    return {"position": e.x, "time": e.time, "momentum": e.pup, "flavor": e.f[:, :e.nh], "flavorbar": e.f[:, e.nh:]}


def exact(case, seed):
    n = case["nx"] * case["ny"] * case["nz"] * case["dirs"]
    width = [1 if m == 1 else case["order"] + 1 for m in (case["nx"], case["ny"], case["nz"])]
    if n * case["steps"] * width[0] * width[1] * width[2] * case["nf"] ** 2 > 8e9:
        return None   # (minutes)
    e = _Exact(case, seed)
    if case["how"] != "adjoint":
        _, m = e.forward(case["steps"])
        out = _out(e)
        if case["how"] == "loop":
            with torch.no_grad():
                out["rate"] = e.rates(e.f, m, e.stencil(e.x))
        if case["mesh"]:
            out["mesh"] = m.t().contiguous()
        return out
    f0, x0, N = e.f.clone().requires_grad_(True), e.x.clone(), e.N.clone().requires_grad_(True)
    dts, _ = e.forward(case["steps"])
    f, x = f0, x0
    for dt in dts:
        f = torch.utils.checkpoint.checkpoint(lambda f, N, x, dt: e.flavor_step(f, N, x, dt)[0], f, N, x, dt,
                                              use_reentrant=False)
        x = e.move(x, dt)
    m = e.deposit(f, N, e.stencil(x))
    k = _re(e.nf, 0, 1)
    J = (m[:, k] ** 2 + m[:, k + 1] ** 2).sum() / e.vol
    gf, gN = torch.autograd.grad(J, (f0, N))
    return {"objective": J.detach(), "grad_flavor": gf, "grad_number": gN, "dts": torch.tensor(dts, dtype=torch.float64)}
