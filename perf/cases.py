"""Performance cases: the calls a filter-diagonalization user makes, as a user makes them.

Every case goes through the public binding (filterbse_gb300.Context, Precond) on systems of
this repository: passivated zincblende CdSe / InP dots on the grids of the reference's grid
rule (workload.py), the 2.2 nm CdSe example (real states, 57 x 52 x 45) and the 1x1x1 CsPbI3
example (spinors, SO + NL projectors, 44^3).  A case is a dict of plain values; `kind` names
the call:

  hpsi     Context.hpsi: one H psi of a batch of states
  filter   Context.newton_filter: a whole Newton filter of a few starts
  range    Context.energy_range: the spectrum range a filter run starts with
  ritz     Context.ortho_diag_sigma: Rayleigh-Ritz of filtered states
  bse      Context.bse_kernel (and bse_solve): the exciton stage
  precond  Precond.apply / Precond.grad: inference and one training gradient

The mixed path computes in single precision but hands some results back as doubles; its
states and energies are returned here at the path's working precision
(Context.working_dtype), the type in which a mixed run hands them on.
"""
from __future__ import annotations

import functools
import math
import os

import numpy as np
import torch

import filterbse_gb300 as F
from filterbse_gb300 import workload as W

GOLDEN = os.path.dirname(W.POT_DIR)
NPROJ = W.NPROJ
DEV = "cuda:0"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _dot(radius, spacing=0.5, extra=(0, 0, 0), material="CdSe", spinor=True, nl=False):
    return {"system": "dot", "material": material, "radius": radius, "spacing": spacing, "extra_x": extra[0],
            "extra_y": extra[1], "extra_z": extra[2], "spinor": spinor, "nl": nl}


EXAMPLE = {"system": "cdse_example", "spinor": False, "nl": False}
PEROVSKITE = {"system": "perovskite", "spinor": True, "nl": True}


def listed():
    return [
        # the batched H psi of the benchmark's 3 nm spinor dot (128^3): most of a production filter run
        {"name": "hpsi_3nm_mixed_16", "kind": "hpsi", "precision": "mixed", "states": 16, **_dot(15.0)},
        # one small real state (the 2.2 nm example's 57 x 52 x 45): a residual check, where latency counts
        {"name": "hpsi_example_mixed_1", "kind": "hpsi", "precision": "mixed", "states": 1, **EXAMPLE},
        # an uneven dot of the multi-dot workload (InP, its own 7-smooth grid, 4 starts)
        {"name": "hpsi_inp_mixed_4", "kind": "hpsi", "precision": "mixed", "states": 4,
         **_dot(12.0, extra=(0, 1, 4), material="InP")},
        # the plain FP64 path a mixed run is judged by, with both projector kinds
        {"name": "hpsi_2nm_fp64_6", "kind": "hpsi", "precision": "fp64", "states": 6, **_dot(10.0, nl=True)},
        # a short mixed filter of a 2 nm dot, 4 starts x 16 targets (the multi-dot workload's batch)
        {"name": "filter_2nm_mixed", "kind": "filter", "precision": "mixed", "states": 4, "targets": 16,
         "ncheby": 128, **_dot(10.0)},
        # the FP64 filter of the real 2.2 nm example: 16 starts x 16 targets
        {"name": "filter_example_fp64", "kind": "filter", "precision": "fp64", "states": 16, "targets": 16,
         "ncheby": 128, **EXAMPLE},
        # the spectrum range of the CsPbI3 cube: hundreds of single H psi with a scalar read after each
        {"name": "range_perovskite_fp64", "kind": "range", "precision": "fp64", "max_iter": 1500, **PEROVSKITE},
        # Rayleigh-Ritz of the real example's filtered states (16 starts x 8 kept targets)
        {"name": "ritz_example_fp64", "kind": "ritz", "precision": "fp64", "states": 128, **EXAMPLE},
        # Rayleigh-Ritz of a mixed spinor run (8 starts x 16 targets, coarse 2.4 nm dot)
        {"name": "ritz_dot_mixed", "kind": "ritz", "precision": "mixed", "states": 128, **_dot(12.0, 0.6)},
        # the electron-hole kernels of a 2 nm dot's 16 holes x 16 electrons
        {"name": "bse_2nm_mixed", "kind": "bse", "precision": "mixed", "holes": 16, "electrons": 16, "solve": False,
         **_dot(10.0)},
        # the whole FP64 exciton stage of the CsPbI3 cube: kernels, then the eigensolve
        {"name": "bse_perovskite_fp64", "kind": "bse", "precision": "fp64", "holes": 14, "electrons": 14,
         "solve": True, **PEROVSKITE},
        # one training gradient of the learned preconditioner on a 1.6 nm dot's residuals
        {"name": "precond_grad", "kind": "precond", "precision": "mixed", "states": 2, "backward": True,
         **_dot(8.0)},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["hpsi", "hpsi", "hpsi", "filter", "filter", "range", "ritz", "ritz", "bse", "bse", "precond"])
    prec = rng.choice(["mixed", "fp64"])
    pick = rng.random()
    if pick < 0.15:
        c = dict(EXAMPLE)
    elif pick < 0.3:
        c = dict(PEROVSKITE)
    else:
        # dots of 0.8 to 2.4 nm at the reference's spacings, grown by up to a dozen points per axis:
        # any parity and any prime factor
        spacing = rng.choice([0.5, 0.6, 0.7, 0.8])
        spinor = rng.random() < 0.7
        c = _dot(round(_log(rng, 4.0, 12.0 if spacing > 0.55 else 10.0), 2), spacing,
                 tuple(rng.randrange(0, 13) for _ in range(3)), rng.choice(["CdSe", "InP"]), spinor,
                 rng.random() < 0.3)
    c |= {"kind": kind, "precision": prec}
    if kind == "hpsi":
        c["states"] = int(_log(rng, 1, 16.9) if prec == "mixed" else _log(rng, 1, 6.9))
    elif kind == "filter":
        c |= {"states": rng.randrange(1, 5), "targets": rng.choice([1, 3, 4, 8, 10, 16]),
              "ncheby": int(_log(rng, 16, 100) if prec == "mixed" else _log(rng, 8, 40))}
    elif kind == "range":
        # the range stops on rounding-sensitive differences of single-precision sums on the mixed path
        c = {"kind": kind, "precision": "fp64", **PEROVSKITE, "max_iter": rng.randrange(40, 1500)}
    elif kind == "ritz":
        c["states"] = int(_log(rng, 3, 129) if prec == "mixed" else _log(rng, 3, 65))
    elif kind == "bse":
        hi = 16.9 if prec == "mixed" else 9.9
        c |= {"holes": int(_log(rng, 1, hi)), "electrons": int(_log(rng, 1, hi)), "solve": rng.random() < 0.5}
        if prec == "mixed":
            c["solve"] = False
        if not c["spinor"]:
            c["solve"] = False
    else:
        c |= {"precision": "mixed", "states": rng.randrange(1, 3), "backward": rng.random() < 0.5}
        if c["system"] == "dot":
            c |= {"radius": min(c["radius"], 8.0)}
    return c


# ---------------------------------------------------------------------------
# systems: grid, local potential and projector table (a user's input files)
# ---------------------------------------------------------------------------

def _read_conf(path):
    with open(path) as f:
        n = int(f.readline())
        rows = [f.readline().split() for _ in range(n)]
    xyz = np.array([[float(v) for v in r[1:4]] for r in rows])
    return [r[0] for r in rows], xyz - xyz.mean(axis=0)


def _projectors(grid, xyz, so_par, nl):
    rc2 = W.r_nlcut2(grid.dx)
    r = np.linspace(0.0, math.sqrt(rc2), W.PROJ_LEN, endpoint=False)
    tab = None
    sgn = np.zeros(len(xyz) * NPROJ, np.int32)
    if nl:  # smooth nonlocal channels of the size of the examples' (NL parameters of 0.01 to 1 Ha)
        one = np.array([0.3 * np.exp(-(r / (0.6 + 0.2 * p)) ** 2) * r / (1.0 + p) for p in range(NPROJ)])
        tab = np.stack([one * (0.8 + 0.1 * (a % 5)) for a in range(len(xyz))])
        sgn = np.where((np.arange(len(xyz) * NPROJ) % 3) == 1, -1, 1).astype(np.int32)
    n_l, npts, jx, y1, sp, nlp = F.build_nlc(grid.axes(), xyz, so_par, W.so_radial(grid.dx, math.sqrt(rc2)), tab,
                                             NPROJ, rc2)
    return W.ProjTable(n_l.astype(np.int64), npts, jx, y1, sp, nlp, sgn, NPROJ)


@functools.lru_cache(maxsize=3)
def _system_of(system, material, radius, spacing, extra_x, extra_y, extra_z, spinor, nl):
    """(grid, potential, projector table or None)"""
    if system == "cdse_example":
        types, xyz = _read_conf(os.path.join(GOLDEN, "cdse22", "conf.par"))
        grid = W.Grid(57, 52, 45, 0.8, 0.8, 0.8, -22.8, -20.8, -18.0, 10.0)
        pots = os.path.join(GOLDEN, "cdse22")
        so = 0.01
    elif system == "perovskite":
        types, xyz = _read_conf(os.path.join(GOLDEN, "cspbi3", "conf.par"))
        grid = W.Grid(44, 44, 44, 0.5, 0.5, 0.5, -11.0, -11.0, -11.0, 20.0)
        pots = os.path.join(GOLDEN, "cspbi3")
        so = {"Pb": 7.79, "I": 2.0, "Cs": 1.0}
    else:
        cat, an, a_ang, pots = W.MATERIALS[material]
        types, xyz = W.zincblende_dot(radius, a_ang, cat, an)
        rule = W.reference_grid(xyz, spacing, 10.0)
        want = (rule.nx + extra_x, rule.ny + extra_y, rule.nz + extra_z)
        grid = W.reference_grid(xyz, spacing, 10.0, n_in=want)
        so = 0.01
    pot = W.local_pot(grid, types, xyz, pots)
    proj = None
    if spinor or nl:
        core = [i for i, t in enumerate(types) if t not in ("P1", "P2")]
        par = np.array([so[types[i]] if isinstance(so, dict) else so for i in core])
        proj = _projectors(grid, xyz[core], par, nl)
    return grid, pot, proj


def _system(case):
    return _system_of(case["system"], case.get("material", ""), case.get("radius", 0.0), case.get("spacing", 0.0),
                      case.get("extra_x", 0), case.get("extra_y", 0), case.get("extra_z", 0), case["spinor"],
                      case["nl"])


def _spins(case):
    return 2 if case["spinor"] else 1


def _context(case):
    grid, pot, proj = _system(case)
    return F.Context(grid, pot, nspin=_spins(case), is_complex=case["spinor"], so=case["spinor"], nl=case["nl"],
                     proj=proj, precision=F.MIXED if case["precision"] == "mixed" else F.FP64)


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _random_states(n, case, gen):
    """n normalised random starts as init_filter_states makes them: uniform on the grid (complex128)"""
    grid = _system(case)[0]
    shape = (n, _spins(case) * grid.ngrid)
    re = torch.rand(shape, dtype=torch.float64, device=DEV, generator=gen) * 2 - 1
    im = torch.rand(shape, dtype=torch.float64, device=DEV, generator=gen) * 2 - 1
    psi = torch.complex(re, im)
    return psi / (torch.linalg.vector_norm(psi, dim=1, keepdim=True) * math.sqrt(grid.dv))


def _smooth_states(n, case, gen):
    """n normalised confined low-energy states: random fields, low-passed, inside an envelope"""
    grid = _system(case)[0]
    psi = _random_states(n, case, gen)
    dims = (grid.nz, grid.ny, grid.nx)
    ks = [torch.fft.fftfreq(m, d, dtype=torch.float64, device=DEV) * 2 * math.pi
          for m, d in zip(dims, (grid.dz, grid.dy, grid.dx))]
    k2 = ks[0][:, None, None] ** 2 + ks[1][None, :, None] ** 2 + ks[2][None, None, :] ** 2
    xs = [(torch.arange(m, dtype=torch.float64, device=DEV) / (m - 1) * 2 - 1) for m in dims]
    env = torch.exp(-3.0 * (xs[0][:, None, None] ** 2 + xs[1][None, :, None] ** 2 + xs[2][None, None, :] ** 2))
    low = torch.exp(-0.5 * k2)
    for row in psi:
        v = row.view(-1, *dims)
        v.copy_(torch.fft.ifftn(torch.fft.fftn(v, dim=(1, 2, 3)) * low, dim=(1, 2, 3)) * env)
    return psi / (torch.linalg.vector_norm(psi, dim=1, keepdim=True) * math.sqrt(grid.dv))


def _stored(psi, case):
    """complex128 states as psitot rows (real jobs keep the real part)"""
    rows = torch.view_as_real(psi).reshape(psi.shape[0], -1) if case["spinor"] else psi.real
    return rows.contiguous()


def _filtered_like(n, case, gen):
    """n overlapping states as a filter leaves them: mixtures of fewer smooth states, so the last tenth
    of the span is dependent up to rounding noise and is cut"""
    rank = max(1, (9 * n) // 10)
    base = _smooth_states(rank, case, gen)
    if not case["spinor"]:
        base = base.real.to(torch.complex128)
    mix = torch.randn((n, rank), dtype=torch.float64, device=DEV, generator=gen)
    if case["spinor"]:
        mix = torch.complex(mix, torch.randn((n, rank), dtype=torch.float64, device=DEV, generator=gen))
    mix = mix.to(torch.complex128)
    return (mix @ base) / math.sqrt(rank)


def _filter_plan(case):
    """(zn, an, vmin, dE) of a short filter: the range from the potential, targets inside the window"""
    grid, pot, _ = _system(case)
    lo = float(pot.min()) - 1.0
    de = float(pot.max()) + grid.ke_max + 2.0 - lo
    zn, _ = F.samp_points(case["ncheby"])
    targets = np.linspace(-0.35, -0.05, case["targets"])
    an = F.newton_coeff(zn, targets, lo, de, (case["ncheby"] / (2.5 * de)) ** 2)
    return zn, an, lo, de


def _bse_inputs(case, seed):
    gen = _gen(seed)
    grid = _system(case)[0]
    nh, ne = case["holes"], case["electrons"]
    psi = _smooth_states(nh + ne, case, gen)
    dims = (grid.nz, grid.ny, grid.nx)
    ks = [torch.fft.fftfreq(m, d, dtype=torch.float64, device=DEV) * 2 * math.pi
          for m, d in zip(dims, (grid.dz, grid.dy, grid.dx))]
    k2 = ks[0][:, None, None] ** 2 + ks[1][None, :, None] ** 2 + ks[2][None, None, :] ** 2
    bare = 4 * math.pi / (k2 + 0.05) / grid.ngrid
    screened = bare / 6.1 * (1.0 + 0.5 * torch.exp(-k2))
    ene = torch.rand(nh + ne, dtype=torch.float64, device=DEV, generator=gen).cpu().numpy() * 0.15
    ene = np.concatenate([np.sort(ene[:nh]) - 0.40, np.sort(ene[nh:]) - 0.10])
    return psi, bare.to(torch.complex128).reshape(-1), screened.to(torch.complex128).reshape(-1), ene


def _ritz_states(case, seed):
    return _stored(_filtered_like(case["states"], case, _gen(seed)), case)


def _hpsi_states(case, seed):
    """working states as hpsi takes them; a real job packs two real states into one"""
    psi = _random_states(case["states"], case, _gen(seed))
    return psi.to(torch.complex64) if case["precision"] == "mixed" else psi


def prepare(case, seed):
    ctx = _context(case)
    kind = case["kind"]
    state = {"case": case, "ctx": ctx}
    if kind == "hpsi":
        state["x"] = _hpsi_states(case, seed)
        state["y"] = torch.empty_like(state["x"])
    elif kind == "filter":
        state["plan"] = _filter_plan(case)
        state["psi0"] = _stored(_random_states(case["states"], case, _gen(seed)), case)
    elif kind == "range":
        state["seed"] = -(874917403 + int(seed) % 1000003)
    elif kind == "ritz":
        state["psi"] = _ritz_states(case, seed)
    elif kind == "bse":
        psi, bare, screened, ene = _bse_inputs(case, seed)
        state |= {"psi": psi if case["spinor"] else psi.real.contiguous(), "bare": bare, "screened": screened,
                  "ene": ene}
    else:
        gen = _gen(seed)
        n = case["states"]
        state["resid"] = torch.randn((n, ctx.stlen), dtype=torch.float64, device=DEV, generator=gen) * 1e-2
        state["corr"] = torch.randn((n, ctx.stlen), dtype=torch.float64, device=DEV, generator=gen) * 1e-3
        state["ene"] = np.linspace(-0.3, -0.1, n)
        state["net"] = F.Precond(ctx, seed=3)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _handed_on(states, ctx):
    """double-typed states of a run at the path's working precision"""
    return states if ctx.working_dtype() is torch.complex128 else states.to(torch.float32)


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "hpsi":
        ctx.hpsi(state["x"], state["y"])
        return state["y"]
    if kind == "filter":
        zn, an, vmin, de = state["plan"]
        return _handed_on(ctx.newton_filter(zn, an, vmin, de, state["psi0"]), ctx)
    if kind == "range":
        emin, emax, iters = ctx.energy_range(state["seed"], case["max_iter"])
        return {"emin": emin, "emax": emax, "iters": iters}
    if kind == "ritz":
        psi = state["psi"].clone()  # the call works in place
        k, ev, sg = ctx.ortho_diag_sigma(psi)
        if case["precision"] == "mixed":
            ev, sg = ev.astype(np.float32), sg.astype(np.float32)
        return {"kept": k, "eval": ev, "sigma": sg, "psi": _handed_on(psi, ctx)}
    if kind == "bse":
        nh, ne = case["holes"], case["electrons"]
        kernel = ctx.bse_kernel if case["spinor"] else ctx.bse_kernel_real
        direct, exchange = kernel(state["psi"], nh, ne, nh, state["bare"], state["screened"])
        if not case["solve"]:
            if case["precision"] == "mixed":
                t = torch.complex64 if case["spinor"] else torch.float32
                direct, exchange = direct.to(t), exchange.to(t)
            return {"direct": direct, "exchange": exchange}
        ene, coeff, h, d, x, h0 = ctx.bse_solve(state["ene"], nh, ne, nh, direct, exchange)
        return {"direct": direct, "exchange": exchange, "ene": ene, "coeff": coeff, "h": h, "d": d, "x": x, "h0": h0}
    if case["backward"]:
        loss, grad = state["net"].grad(state["resid"], state["corr"], state["ene"])
        return {"loss": loss, "grad": grad}
    return state["net"].apply(state["resid"], state["ene"])


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------

def _ls():
    """L.S in the flattened (spin, m) basis, row j' = 3 s' + m', column j = 3 s + m"""
    h = math.sqrt(0.5)
    lx = np.array([[0, h, 0], [h, 0, h], [0, h, 0]], complex)
    ly = 1j * np.array([[0, h, 0], [-h, 0, h], [0, -h, 0]])
    lz = np.diag([-1.0, 0.0, 1.0]).astype(complex)
    sx = np.array([[0, 0.5], [0.5, 0]], complex)
    sy = 1j * np.array([[0, -0.5], [0.5, 0]])
    sz = np.diag([0.5, -0.5]).astype(complex)
    return sum(np.kron(s.T, l.T) for l, s in ((lx, sx), (ly, sy), (lz, sz)))


class _Hamiltonian:
    def __init__(self, case):
        grid, pot, proj = _system(case)
        self.spins, self.grid = _spins(case), grid
        self.dims = (grid.nz, grid.ny, grid.nx)
        dk = grid.dk()
        k2 = []
        for n, d in zip((grid.nx, grid.ny, grid.nz), dk):
            j = torch.arange(n, device=DEV)
            k2.append(0.5 * (torch.minimum(j, n - j).double() * d) ** 2)
        self.kin = (k2[2][:, None, None] + k2[1][None, :, None] + k2[0][None, None, :]).clamp(max=grid.ke_max)
        self.pot = torch.tensor(pot, device=DEV)
        self.proj = []
        if proj is not None:
            nat, npts = len(proj.nl), int(proj.npts)
            live = torch.arange(npts, device=DEV)[None, :] < torch.tensor(proj.nl, device=DEV)[:, None]
            self.j = torch.where(live, torch.tensor(proj.jxyz, device=DEV).reshape(nat, npts).long(), 0)
            y = torch.tensor(np.ascontiguousarray(proj.y1), device=DEV).reshape(nat, npts, 3, 2)
            self.y = torch.where(live[..., None], torch.complex(y[..., 0], y[..., 1]), 0)
            radial = lambda v: torch.where(live[..., None], torch.tensor(np.ascontiguousarray(v), device=DEV)  # noqa: E731
                                           .reshape(nat, npts, NPROJ), 0).to(torch.complex128)
            if case["spinor"]:
                self.proj.append((radial(proj.proj), torch.tensor(_ls(), device=DEV), None))
            if case["nl"]:
                sgn = torch.tensor(proj.sgn.reshape(nat, NPROJ, 1), device=DEV).to(torch.complex128)
                self.proj.append((radial(proj.nlp), None, sgn))

    def __call__(self, psi):
        """H psi of [n, spins * ngrid] complex128 states"""
        out = torch.empty_like(psi)
        for row, o in zip(psi, out):
            v = row.view(self.spins, *self.dims)
            t = torch.fft.ifftn(torch.fft.fftn(v, dim=(1, 2, 3)) * self.kin, dim=(1, 2, 3))
            o.copy_((t.reshape(self.spins, -1) + row.view(self.spins, -1) * self.pot).reshape(-1))
            for rad, ls, sgn in self.proj:
                at = row.view(self.spins, -1)[:, self.j]  # [spins, atoms, points]
                terms = at.permute(1, 2, 0)[..., None] * self.y.conj()[:, :, None, :]
                c = self.grid.dv * rad.transpose(1, 2) @ terms.reshape(*self.j.shape, 3 * self.spins)
                c = c @ ls if ls is not None else c * sgn
                back = (rad @ c).reshape(*self.j.shape, self.spins, 3) * self.y[:, :, None, :]
                back = back.sum(-1).permute(2, 0, 1).reshape(self.spins, -1)
                for s in range(self.spins):
                    o.view(self.spins, -1)[s].index_add_(0, self.j.reshape(-1), back[s])
        return out


def _exact_filter(case, seed):
    ham = _Hamiltonian(case)
    zn, an, vmin, de = _filter_plan(case)
    an = torch.tensor(an.real, device=DEV)
    psi = _random_states(case["states"], case, _gen(seed))
    if not case["spinor"]:
        psi = psi.real.to(torch.complex128)
    if case["precision"] == "mixed":
        psi = psi.to(torch.complex64).to(torch.complex128)
    out = torch.zeros((psi.shape[0], case["targets"], psi.shape[1]), dtype=torch.complex128, device=DEV)
    for j in range(len(zn)):
        if j:
            psi = 4.0 / de * ham(psi) - (2.0 + zn[j - 1] + 4.0 / de * vmin) * psi
        for t in range(case["targets"]):
            out[:, t] += an[t, j] * psi
    rows = torch.view_as_real(out).reshape(out.shape[0], out.shape[1], -1) if case["spinor"] else out.real
    return rows.contiguous()


def _exact_ritz(case, seed):
    ham = _Hamiltonian(case)
    dv = ham.grid.dv
    rows = _ritz_states(case, seed)
    psi = torch.view_as_complex(rows.view(rows.shape[0], -1, 2)) if case["spinor"] else rows.to(torch.complex128)
    hpsi = ham(psi)
    over = dv * (psi.conj() @ psi.T)
    proj = dv * (psi.conj() @ hpsi.T)
    lam, vec = np.linalg.eigh(over.cpu().numpy())
    keep = lam > lam.max() * (1e-6 if case["precision"] == "mixed" else 1e-12)
    x = vec[:, keep] / np.sqrt(lam[keep])
    h = x.conj().T @ proj.cpu().numpy() @ x
    ev, u = np.linalg.eigh((h + h.conj().T) / 2)
    coef = torch.tensor(x @ u, device=DEV)
    r = coef.T @ hpsi - torch.tensor(ev, device=DEV)[:, None] * (coef.T @ psi)
    sigma = torch.linalg.vector_norm(r, dim=1).cpu().numpy() * math.sqrt(dv)
    return {"kept": None, "eval": ev, "sigma": sigma, "psi": None}


def _exact_bse(case, seed):
    grid = _system(case)[0]
    nh, ne, dims = case["holes"], case["electrons"], (grid.nz, grid.ny, grid.nx)
    psi, bare, screened, ene = _bse_inputs(case, seed)
    if not case["spinor"]:
        psi = psi.real.to(torch.complex128)
    psi = psi.view(nh + ne, _spins(case), -1)
    hole, elec = psi[:nh], psi[nh:]

    def density(a, b):  # rho[x, y] = sum over spins of conj(a_x) b_y
        return torch.stack([(a[x].conj()[None] * b).sum(1) for x in range(a.shape[0])])

    def convolve(rho, pot):
        for row in rho:
            v = row.view(-1, *dims)
            f = torch.fft.fftn(v, dim=(1, 2, 3)) * pot.view(dims) * grid.ngrid
            v.copy_(torch.fft.ifftn(f, dim=(1, 2, 3)))
        return rho

    # direct[(a,i),(b,j)] = dv sum [W rho_ab] rho_ji, exchange = -dv sum [v rho_ai] rho_jb
    p = convolve(density(elec, elec), screened).reshape(ne * ne, -1)
    q = density(hole, hole).reshape(nh * nh, -1)
    direct = (grid.dv * p @ q.T).reshape(ne, ne, nh, nh).permute(0, 3, 1, 2).reshape(ne * nh, ne * nh)
    p = convolve(density(elec, hole), bare).reshape(ne * nh, -1)
    q = density(hole, elec).transpose(0, 1).reshape(ne * nh, -1)
    exchange = -grid.dv * p @ q.T
    if not case["spinor"]:
        direct, exchange = direct.real, 2 * exchange.real
    direct, exchange = torch.tril(direct), torch.tril(exchange)
    if not case["solve"]:
        return {"direct": direct, "exchange": exchange}

    def full(m):
        low = torch.tril(m, -1)
        return low + low.conj().T + torch.diag(torch.diag(m).real).to(m.dtype)

    direct, exchange = full(direct), full(exchange)
    h0 = torch.tensor((ene[nh:, None] - ene[None, :nh]).reshape(-1), device=DEV)
    ham = torch.diag(h0).to(torch.complex128) - direct - exchange
    ev, u = np.linalg.eigh(ham.cpu().numpy())
    u = torch.tensor(u, device=DEV)
    mean = lambda m: (u.conj() * (m @ u)).sum(0).real  # noqa: E731
    return {"direct": direct, "exchange": exchange, "ene": ev, "coeff": None, "h": mean(ham), "d": mean(direct),
            "x": mean(exchange), "h0": mean(torch.diag(h0).to(torch.complex128))}


def exact(case, seed):
    kind = case["kind"]
    if kind == "hpsi":
        return _Hamiltonian(case)(_hpsi_states(case, seed).to(torch.complex128))
    if kind == "filter":
        return _exact_filter(case, seed)
    if kind == "ritz":
        return _exact_ritz(case, seed)
    if kind == "bse":
        return _exact_bse(case, seed)
    return None  # the range is where an iteration stops; the network rounds its activations to BF16


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    grid, _, proj = _system(case)
    n, spins = grid.ngrid, _spins(case)
    val = 4 if case["precision"] == "mixed" else 8  # bytes of a working value
    entries = int(np.sum(proj.nl)) if proj is not None else 0
    channels = (1 if case["spinor"] else 0) + (1 if case["nl"] else 0)
    fft = 5.0 * n * math.log2(n)  # flops of one transform of one block
    # per state: two transforms, kinetic factor, V and the shift; the projector sums both ways
    h_flops = spins * (2 * fft + 10.0 * n) + entries * channels * spins * (78 + 84)
    tables = n * val + entries * (4 + 6 * val + channels * NPROJ * val)
    stlen = spins * n * (2 if case["spinor"] else 1)
    kind = case["kind"]
    if kind == "hpsi":
        s = case["states"]
        return {"bytes": 2.0 * s * spins * n * 2 * val + tables, "flops": s * h_flops}
    if kind == "filter":
        s, m, k = case["states"], case["targets"], case["ncheby"]
        states = s if case["spinor"] else (s + 1) // 2  # two real states share one complex one
        return {"bytes": 8.0 * s * (1 + m) * stlen + tables, "flops": states * (k - 1) * h_flops + 2.0 * k * m * s * stlen}
    if kind == "range":
        return {"bytes": float(tables), "flops": 2 * h_flops}  # the iteration count is the system's
    if kind == "ritz":
        s = case["states"]
        cplx = 8.0 if case["spinor"] else 2.0
        return {"bytes": 16.0 * s * stlen + tables,
                "flops": s * h_flops + cplx * spins * n * (s * (s + 1.0) + 2.0 * s * s)}
    if kind == "bse":
        nh, ne = case["holes"], case["electrons"]
        x = nh * ne
        cplx = 8.0 if case["spinor"] else 2.0
        out = 16.0 if case["spinor"] else 8.0
        flops = (ne * ne + x) * 2 * fft + cplx * n * x * (x + 1.0)  # the kept triangles of both kernels
        return {"bytes": out * (nh + ne) * spins * n + 32.0 * n + 2 * out * x * x,
                "flops": flops + (25 * 4.0 * x ** 3 if case["solve"] else 0.0)}
    fields = case["states"] * stlen // n
    passes = 3 if case["backward"] else 1
    return {"bytes": 8.0 * case["states"] * stlen * 2 + 4.0 * n, "flops": passes * 2.0 * F.PRECOND_NWEIGHTS * n * fields}
