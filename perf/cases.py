"""The work that a user of this library has it do, as cases that can be timed.

Every case goes through the public methods of `cvc_b200.Lattice` on fields in
GPU memory.  The lattices are those of the repository's tests, benchmark and
configurations (8 x 4^3 up to 64 x 32^3) and, among the drawn cases, extents of
no particular form.  The families:

  op        one application of the twisted-mass operator (Q_phi_tbc, Q_phi,
            Qf5, Hopping) to a field
  bicgstab  one propagator column by the FP64 BiCGStab of invert_Qtm_her
  solve     propagator columns by the batched mixed-precision solver
  contract  Pi_mu_nu(x) of one source point from its 120 columns
  adjoint   Pi_mu_nu(x) with its gradients in the twisted mass, the hopping
            parameter and the gauge links: forward and backward pass
  momentum  Pi_mu_nu(q) from Pi_mu_nu(x)

`exact` restates each of them in plain torch with 64-bit arithmetic.
"""
import math

import numpy as np
import torch

import cvc_b200

PRECISION = {"double": cvc_b200.PREC_DOUBLE, "single": cvc_b200.PREC_SINGLE,
             "half": cvc_b200.PREC_HALF}


def listed():
    return [
        # the smallest lattice of the tests: what one operator call costs by itself
        dict(name="op_8x4x4x4", kind="op", op="Q_phi_tbc", T=8, LX=4, LY=4, LZ=4),
        # no extent alike, none a multiple of a warp: an ordinary call of odd form
        dict(name="op_22x14x10x18", kind="op", op="Qf5", T=22, LX=14, LY=10, LZ=18),
        # the largest configuration: a residual check of one column
        dict(name="op_64x32x32x32", kind="op", op="Q_phi_tbc", T=64, LX=32, LY=32, LZ=32),
        # one column by the solver that keeps the reference's algorithm
        dict(name="bicgstab_32x16x16x16", kind="bicgstab", T=32, LX=16, LY=16, LZ=16, kappa=0.150,
             mu2k=0.01, eps=0.3, precision2=1e-24),
        # a single column on a small lattice: launches and checks count (the tmLQCD
        # interface hands over one column per call)
        dict(name="solve_16x8x8x8_n1", kind="solve", T=16, LX=8, LY=8, LZ=8, kappa=0.150, mu2k=0.01,
             eps=0.3, columns=1, source="point", precision="single", tol=1e-10),
        # the 12 columns of a source point with FP16 storage in the inner iterations
        dict(name="solve_32x16x16x16_n12_half", kind="solve", T=32, LX=16, LY=16, LZ=16, kappa=0.150,
             mu2k=0.01, eps=0.3, columns=12, source="point", precision="half", tol=1e-10),
        # the 12 columns of a source point at the benchmark's configuration
        dict(name="solve_48x24x24x24_n12", kind="solve", T=48, LX=24, LY=24, LZ=24, kappa=0.155,
             mu2k=0.005, eps=0.25, columns=12, source="point", precision="single", tol=1e-10),
        # the benchmark: 8 source points
        dict(name="solve_48x24x24x24_n96", kind="solve", T=48, LX=24, LY=24, LZ=24, kappa=0.155,
             mu2k=0.005, eps=0.25, columns=96, source="point", precision="single", tol=1e-10),
        # a small contraction: 120 fields of 1.6 MB
        dict(name="contract_16x8x8x8", kind="contract", T=16, LX=8, LY=8, LZ=8),
        # the contraction of the benchmark's configuration
        dict(name="contract_48x24x24x24", kind="contract", T=48, LX=24, LY=24, LZ=24),
        # the configuration that the derivatives are quoted on
        dict(name="adjoint_24x12x12x12", kind="adjoint", T=24, LX=12, LY=12, LZ=12, kappa=0.150,
             mu2k=0.01, eps=0.3, precision="single", tol=1e-12),
        # the Fourier transform after the contraction
        dict(name="momentum_48x24x24x24", kind="momentum", T=48, LX=24, LY=24, LZ=24),
    ]


# Largest volumes of the drawn cases, at most the listed ones'.
_CAP = {"op": 64 * 32 ** 3, "bicgstab": 32 * 16 ** 3, "contract": 48 * 24 ** 3,
        "adjoint": 24 * 12 ** 3, "momentum": 48 * 24 ** 3}


def _extents(rng, largest):
    """Four even extents whose volume is spread evenly over its logarithm."""
    want = math.exp(rng.uniform(math.log(512), math.log(largest)))
    while True:
        side = [max(2, round(want ** 0.25 * math.exp(rng.uniform(-0.6, 0.6)) / 2)) * 2 for _ in range(4)]
        if 0.7 * want <= math.prod(side) <= min(1.3 * want, largest):
            return dict(zip(("T", "LX", "LY", "LZ"), side))


def draw(rng):
    kind = rng.choice(["op", "op", "bicgstab", "solve", "solve", "solve", "contract", "contract",
                       "adjoint", "momentum"])
    if kind == "op":
        return dict(kind=kind, op=rng.choice(["Q_phi_tbc", "Q_phi", "Qf5", "Hopping"]),
                    **_extents(rng, _CAP[kind]))
    if kind in ("contract", "momentum"):
        return dict(kind=kind, **_extents(rng, _CAP[kind]))
    c = dict(kind=kind, kappa=rng.choice([0.140, 0.150]), mu2k=rng.choice([0.01, 0.02]),
             eps=rng.choice([0.25, 0.3]))
    if kind == "bicgstab":
        return dict(c, precision2=1e-24, **_extents(rng, _CAP[kind]))
    if kind == "adjoint":
        return dict(c, precision="single", tol=1e-12, **_extents(rng, _CAP[kind]))
    n = rng.choice([1, 2, 5, 12, 17, 24, 48, 60, 96])
    return dict(c, columns=n, source=rng.choice(["point", "timeslice"]),
                precision=rng.choice(["single", "single", "half", "double"]), tol=1e-10,
                **_extents(rng, min(32 * 16 ** 3, 96 * 32 * 16 ** 3 // n)))


# ---- inputs -----------------------------------------------------------------
def _dims(case):
    return case["T"], case["LX"], case["LY"], case["LZ"]


def _volume(case):
    return math.prod(_dims(case))


def _mu(case):
    return case.get("mu2k", 0.01) / (2 * case.get("kappa", 0.150))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _gell_mann():
    m = torch.zeros(8, 3, 3, dtype=torch.complex128)
    for a, (i, j) in enumerate([(0, 1), (0, 2), (1, 2)]):
        m[2 * a, i, j] = m[2 * a, j, i] = 1
        m[2 * a + 1, i, j], m[2 * a + 1, j, i] = -1j, 1j
    m[6, 0, 0], m[6, 1, 1] = 1, -1
    m[7] = torch.diag(torch.tensor([1, 1, -2], dtype=torch.complex128)) / math.sqrt(3)
    return m.cuda()


def _gauge(case, gen):
    """Links exp(i eps H), H = sum_a w_a lambda_a / 2 with normal w_a: the
    recipe of the benchmark's gauge field.  Complex [V, 4, 3, 3]."""
    V = _volume(case)
    lam = _gell_mann().reshape(8, 9)
    out = torch.empty(4 * V, 3, 3, dtype=torch.complex128, device="cuda")
    for part in out.split(1 << 20):  # the exponential's work space stays small
        w = torch.randn(len(part), 8, dtype=torch.float64, device="cuda", generator=gen)
        h = (0.5j * case.get("eps", 0.3) * w).to(torch.complex128) @ lam
        part.copy_(torch.linalg.matrix_exp(h.reshape(-1, 3, 3)))
    return out.reshape(V, 4, 3, 3)


def _flat(z):
    return torch.view_as_real(z.contiguous()).reshape(-1)


def _decay(case, site):
    """exp(-distance / 2) from a site, per site: how a propagator falls off."""
    d2 = torch.zeros((), dtype=torch.float64, device="cuda")
    for m, (n, y) in enumerate(zip(_dims(case), np.unravel_index(site, _dims(case)))):
        k = (torch.arange(n, device="cuda", dtype=torch.float64) - int(y)).abs()
        k = torch.minimum(k, n - k)
        shape = [1] * 4
        shape[m] = n
        d2 = d2 + (k * k).reshape(shape)
    return torch.exp(-0.5 * d2.sqrt()).reshape(-1)


def _inputs(case, seed):
    """Everything a case reads, from the seed alone."""
    gen, V, kind = _generator(seed), _volume(case), case["kind"]
    rand = lambda *n: torch.randn(*n, dtype=torch.float64, device="cuda", generator=gen)  # noqa: E731
    site = int(torch.randint(V, (1,), device="cuda", generator=gen))
    d = {"site": site}
    if kind != "momentum":
        d["gauge"] = _gauge(case, gen)
    if kind == "op":
        d["phi"] = rand(24 * V)
    elif kind == "bicgstab":
        d["phi"] = torch.zeros(24 * V, dtype=torch.float64, device="cuda")
        d["phi"][24 * site + 2 * (seed % 12)] = 1.0
    elif kind == "solve":
        b = torch.zeros(case["columns"], 24 * V, dtype=torch.float64, device="cuda")
        if case["source"] == "point":  # 12 spin-colour columns per source point
            at = torch.randint(V, (-(-len(b) // 12),), device="cuda", generator=gen).tolist()
            for i in range(len(b)):
                b[i, 24 * at[i // 12] + 2 * (i % 12)] = 1.0
        else:  # a timeslice of a propagator, as a sequential source has it
            s = 24 * V // case["T"]
            t = int(torch.randint(case["T"], (1,), device="cuda", generator=gen))
            b[:, t * s:(t + 1) * s] = 0.1 * rand(len(b), s)
        d["b"] = b
    elif kind == "contract":
        fall = _decay(case, site).reshape(1, V, 1)
        f = torch.empty(120, V, 24, dtype=torch.float64, device="cuda")
        for part in f.split(12):
            part.copy_(0.2 * fall * rand(*part.shape))
        d["fields"] = f.reshape(120, 24 * V)
    elif kind == "momentum":
        d["conn"] = (0.05 * _decay(case, site).reshape(V, 1) ** 2 * rand(V, 32)).reshape(-1)
        d["contact"] = 0.5 * rand(8)
    elif kind == "adjoint":  # a cosine in z on every (mu, nu), as a momentum projection has it
        z = torch.arange(V, device="cuda") % case["LZ"]
        d["w"] = (torch.cos(2 * math.pi * z / case["LZ"]).reshape(V, 1) * rand(1, 32)).reshape(-1)
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    d["case"] = case
    lat = cvc_b200.Lattice(*_dims(case), kappa=case.get("kappa", 0.150), mu=_mu(case))
    V, kind = lat.VOLUME, case["kind"]
    torch.cuda.synchronize()
    if "gauge" in d:
        lat.upload_gauge(_flat(d.pop("gauge")))
    new = lambda *n: torch.zeros(*n, dtype=torch.float64, device="cuda")  # noqa: E731
    if kind in ("op", "bicgstab"):
        d["xi"] = new(24 * V)
    elif kind == "solve":
        d["x"] = new(case["columns"], 24 * V)
    elif kind in ("contract", "momentum"):
        d["out"] = new(32 * V)
        if kind == "momentum":
            d["contact"] = d["contact"].cpu().numpy()
    elif kind == "adjoint":
        d["w"] = d["w"].cpu().numpy()
    if kind in ("solve", "adjoint"):
        p = cvc_b200.solver_defaults()
        p.precision, p.tol = PRECISION[case["precision"]], case["tol"]
        d["params"] = p
    d["lat"] = lat
    return d


def run(state):
    case, lat = state["case"], state["lat"]
    kind = case["kind"]
    if kind == "op":
        op = getattr(lat, case["op"])
        if case["op"] in ("Qf5", "Q_phi"):
            op(state["xi"], state["phi"], -lat.g_mu)
        else:
            op(state["xi"], state["phi"])
        return state["xi"]
    if kind == "bicgstab":
        # the start guess is zero; the library works on its own stream, so the
        # field has to be written before the call
        state["xi"].zero_()
        torch.cuda.current_stream().synchronize()
        n = lat.invert_Qtm_her(state["xi"], state["phi"], case["precision2"], 5000)
        if n < 0:
            raise RuntimeError(f"invert_Qtm_her returned {n}")
        return state["xi"]
    if kind == "solve":
        x, b = state["x"], state["b"]
        st = lat.solve(list(x), list(b), state["params"])
        if st.converged != len(x):
            raise RuntimeError(f"{len(x) - st.converged} columns did not converge")
        return list(x.split(12))
    if kind == "contract":
        conn, contact = lat.cvc_contract(list(state["fields"]), state["site"], conn=state["out"])
        return {"conn": conn, "contact": contact}
    if kind == "momentum":
        return lat.pi_momentum(state["conn"], state["site"], state["contact"], out=state["out"])
    conn, contact = lat.pi_forward(state["site"], state["params"])
    dmu, dkappa, dgauge = lat.pi_backward(state["w"])
    return {"conn": conn, "contact": contact, "dmu": dmu, "dkappa": dkappa, "dgauge": dgauge}


# Iterations that the solves of the configurations take (measured; they hardly
# depend on the volume): invert_Qtm_her, and conjugate gradients on the
# even/odd preconditioned normal equations.
_HER_ITERATIONS, _CG_ITERATIONS = 100, 40
_OP_FLOPS = 1392  # per site: 8 projected hops and the diagonal


def work(case):
    """Compulsory bytes (inputs once, outputs once) and operations of a pass."""
    V, kind = _volume(case), case["kind"]
    links = 4 * 144 * V
    if kind == "op":
        return {"bytes": links + 2 * 192 * V, "flops": _OP_FLOPS * V}
    if kind == "bicgstab":
        return {"bytes": links + 2 * 192 * V, "flops": _HER_ITERATIONS * 4 * _OP_FLOPS * V}
    if kind == "solve":
        n = case["columns"]
        return {"bytes": links + n * 2 * 192 * V, "flops": n * _CG_ITERATIONS * 2 * _OP_FLOPS * V}
    # per site: 4 nu, 24 columns, 4 mu: two half-spinor hops (2 x 156) and two
    # dots (2 x 48), and the coefficient sums of the dn columns
    pi = 4 * 24 * (4 * (2 * 156 + 2 * 48) + 6 * 12 * 8) * V
    if kind == "contract":
        return {"bytes": links + 120 * 192 * V + 256 * V, "flops": pi}
    if kind == "adjoint":  # 240 columns; the backward pass has three such contractions
        return {"bytes": 2 * links + 3 * 256 * V, "flops": 240 * _CG_ITERATIONS * 2 * _OP_FLOPS * V + 4 * pi}
    return {"bytes": 2 * 256 * V, "flops": 5 * 16 * V * math.log2(V)}


# ---- the same in plain torch, 64 bits ----------------------------------------
def _gammas():
    g = torch.zeros(4, 4, 4, dtype=torch.complex128)
    for k, v in {(0, 0, 2): -1, (0, 1, 3): -1, (0, 2, 0): -1, (0, 3, 1): -1,
                 (1, 0, 3): -1j, (1, 1, 2): -1j, (1, 2, 1): 1j, (1, 3, 0): 1j,
                 (2, 0, 3): -1, (2, 1, 2): 1, (2, 2, 1): 1, (2, 3, 0): -1,
                 (3, 0, 2): -1j, (3, 1, 3): 1j, (3, 2, 0): 1j, (3, 3, 1): -1j}.items():
        g[k] = v
    return g.to(_device())


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


_G5 = (1.0, 1.0, -1.0, -1.0)


class _Wilson:
    """The operator on complex fields [columns, V, 4 spins, 3 colours]; U are
    the links [V, 4, 3, 3] without the boundary phase (antiperiodic in time)."""

    def __init__(self, dims, U):
        self.dims = dims
        self.gamma = _gammas()
        self.g5 = torch.tensor(_G5, dtype=torch.float64, device=U.device).reshape(4, 1)
        phase = torch.ones(4, dtype=torch.complex128, device=U.device)
        phase[0] = complex(math.cos(math.pi / dims[0]), math.sin(math.pi / dims[0]))
        self.W = U * phase.reshape(4, 1, 1)

    def shift(self, f, mu, by):
        """g(x) = f(x + by mu) for a field [columns, V, ...]."""
        lat = f.reshape(f.shape[0], *self.dims, *f.shape[2:])
        return torch.roll(lat, -by, 1 + mu).reshape(f.shape)

    def link(self, mu, f):
        return torch.einsum("xij,cxsj->cxsi", self.W[:, mu], f)

    def link_dagger(self, mu, f):
        return torch.einsum("xji,cxsj->cxsi", self.W[:, mu].conj(), f)

    def spin(self, m, f):
        return torch.einsum("st,cxti->cxsi", m, f)

    def projected(self, mu, sign, f):
        """(1 + sign gamma_mu) f."""
        return f + sign * self.spin(self.gamma[mu], f)

    def hop(self, f):
        out = torch.zeros_like(f)
        for mu in range(4):
            out = out + self.link(mu, self.projected(mu, -1, self.shift(f, mu, 1)))
            out = out + self.shift(self.link_dagger(mu, self.projected(mu, 1, f)), mu, -1)
        return out

    def Q(self, f, kappa, mu):
        return f / (2 * kappa) + 1j * mu * self.g5 * f - 0.5 * self.hop(f)

    def solve(self, b, kappa, mu, tol=1e-14):
        """Q(mu)^-1 b by conjugate gradients on Q^+ Q, all columns at once."""
        Qd = lambda f: self.g5 * self.Q(self.g5 * f, kappa, -mu)  # noqa: E731
        norm = lambda f: f.abs().square().sum((1, 2, 3), keepdim=True)  # noqa: E731
        x, r0 = torch.zeros_like(b), norm(b)
        r0 = torch.where(r0 > 0, r0, torch.ones_like(r0))
        for _ in range(3):  # restarts from the recomputed residual
            res = b - self.Q(x, kappa, mu)
            if float((norm(res) / r0).max()) < tol * tol:
                break
            r = Qd(res)
            p, rr = r.clone(), norm(r)
            stop = rr * 1e-20 + 1e-300
            for k in range(3000):
                q = self.Q(p, kappa, mu)
                a = rr / norm(q).clamp_min(1e-300)
                x += a * p
                r -= a * Qd(q)
                new = norm(r)
                p = r + (new / rr.clamp_min(1e-300)) * p
                rr = new
                if k % 10 == 9 and bool((rr < stop).all()):
                    break
        return x


def _complex(flat, n, V):
    return torch.view_as_complex(flat.reshape(n, V, 4, 3, 2))


def _vertex(w, nu):
    """gamma_nu gamma_5 as the source vertex has it."""
    return w.gamma[nu] @ torch.diag(w.g5.reshape(4)).to(torch.complex128)


def _pi(w, up, dn, site):
    """Pi_mu_nu(x) as complex [V, 4, 4] from columns [60, V, 4, 3], column
    12 m + 3 spin + colour of the source at site + m (m = 4: at the site)."""
    g5 = torch.diag(w.g5.reshape(4)).to(torch.complex128)
    rows = []
    for nu in range(4):
        us = w.W[site, nu]
        pi = [0.0] * 4
        for part in range(2):
            m, n = (4, nu) if part == 0 else (nu, 4)
            phi, chi = up[12 * m:12 * m + 12], dn[12 * n:12 * n + 12]
            spin = _vertex(w, nu) + (g5 if part else -g5)
            colour = us if part == 0 else us.conj().T.resolve_conj().contiguous()
            z = torch.einsum("cd,dxsi->cxsi", torch.kron(spin, colour).conj(), chi)
            for mu in range(4):
                f = -w.g5 * w.link(mu, w.projected(mu, -1, w.shift(phi, mu, 1)))
                b = w.g5 * w.link_dagger(mu, w.projected(mu, 1, phi))
                pi[mu] = pi[mu] + (z.conj() * f).sum((0, 2, 3)) + (w.shift(z, mu, 1).conj() * b).sum((0, 2, 3))
        rows.append(torch.stack(pi, 1))
    return -0.25 * torch.stack(rows, 2)


def _contact(w, up, site, dims):
    out = torch.zeros(4, dtype=torch.complex128, device=up.device)
    at = np.unravel_index(site, dims)
    for nu in range(4):
        to = list(at)
        to[nu] = (to[nu] + 1) % dims[nu]
        far = int(np.ravel_multi_index(to, dims))
        us, one = w.W[site, nu], torch.eye(4, dtype=torch.complex128, device=up.device)
        # trace over spin and colour of (gamma - 1) U S(y + nu, y) and (gamma + 1) U^+ S(y, y + nu)
        s0 = torch.einsum("ij,csj->csi", us, up[48:60, far])
        s1 = torch.einsum("ij,csj->csi", us.conj().T, up[12 * nu:12 * nu + 12, site])
        t0 = torch.einsum("st,cti->csi", w.gamma[nu] - one, s0).reshape(12, 12)
        t1 = torch.einsum("st,cti->csi", w.gamma[nu] + one, s1).reshape(12, 12)
        out[nu] = -0.5 * t0.diagonal().sum() + 0.5 * t1.diagonal().sum()
    return out


def _point_columns(case, site):
    V, dims = _volume(case), _dims(case)
    b = torch.zeros(60, V, 12, dtype=torch.complex128, device=_device())
    for m in range(5):
        at = list(np.unravel_index(site, dims))
        if m < 4:
            at[m] = (at[m] + 1) % dims[m]
        for k in range(12):
            b[12 * m + k, int(np.ravel_multi_index(at, dims)), k] = 1.0
    return b.reshape(60, V, 4, 3)


def _exact_adjoint(case, d):
    dims, V, site = _dims(case), _volume(case), d["site"]
    weights = torch.view_as_complex(d["w"].reshape(V, 4, 4, 2))
    kappa, mu = case["kappa"], _mu(case)
    w = _Wilson(dims, d["gauge"])
    b = _point_columns(case, site)
    up, dn = w.solve(b, kappa, mu), w.solve(b, kappa, -mu)
    U = d["gauge"].clone().requires_grad_(True)
    up.requires_grad_(True), dn.requires_grad_(True)
    pi = _pi(_Wilson(dims, U), up, dn, site)
    (weights.conj() * pi).real.sum().backward()
    dU = U.grad
    km = torch.tensor([kappa, mu], dtype=torch.float64, device=U.device, requires_grad=True)
    for cols, sign in ((up, 1), (dn, -1)):  # lambda = Q^-dagger (dL/dcolumn)
        lam = w.g5 * w.solve(w.g5 * cols.grad, kappa, -sign * mu)
        for at in range(0, 60, 12):
            U2 = d["gauge"].clone().requires_grad_(True)
            q = _Wilson(dims, U2).Q(cols.detach()[at:at + 12], km[0], sign * km[1])
            (-(lam[at:at + 12].conj() * q).real.sum()).backward()
            dU = dU + U2.grad
    return {"conn": _flat(pi.detach()), "contact": _flat(_contact(w, up.detach(), site, dims)),
            "dmu": float(km.grad[1]), "dkappa": float(km.grad[0]), "dgauge": _flat(dU)}


def exact(case, seed):
    V, kind, dims = _volume(case), case["kind"], _dims(case)
    if kind == "solve" and V * case["columns"] > 12 * 48 * 24 ** 3:
        return None  # takes minutes
    d = _inputs(case, seed)
    kappa, mu = case.get("kappa", 0.150), _mu(case)
    if kind == "momentum":
        f = torch.view_as_complex(d["conn"].reshape(*dims, 4, 4, 2))
        f = torch.fft.fftn(f, dim=(0, 1, 2, 3))
        q = [2 * math.pi * torch.arange(n, dtype=torch.float64, device=f.device) / n for n in dims]
        grid = torch.meshgrid(*q, indexing="ij")
        y = np.unravel_index(d["site"], dims)
        qy = sum(g * int(c) for g, c in zip(grid, y))
        for m in range(4):
            for n in range(4):
                f[..., m, n] *= torch.exp(1j * (qy - 0.5 * grid[m] + 0.5 * grid[n]))
                if m == n:
                    f[..., m, n] -= complex(d["contact"][2 * n], d["contact"][2 * n + 1])
        return _flat(f)
    if kind == "adjoint":
        return _exact_adjoint(case, d)
    w = _Wilson(dims, d["gauge"])
    if kind == "op":
        f = _complex(d["phi"], 1, V)
        if case["op"] == "Hopping":
            return _flat(-kappa * w.hop(f))
        r = w.Q(f, kappa, mu if case["op"] == "Q_phi_tbc" else -mu)
        return _flat(w.g5 * r if case["op"] == "Qf5" else r)
    if kind == "bicgstab":
        return _flat(w.solve(_complex(d["phi"], 1, V), kappa, mu))
    if kind == "solve":
        return [torch.cat([_flat(w.solve(_complex(col, 1, V), kappa, mu)) for col in part]).reshape(len(part), -1)
                for part in d["b"].split(12)]
    cols = _complex(d["fields"], 120, V)
    return {"conn": _flat(_pi(w, cols[:60], cols[60:], d["site"])),
            "contact": _flat(_contact(w, cols[:60], d["site"], dims))}
