"""The work that users of this package have it do, as cases that can be timed.

A case is one pass through the public entry points: the Python classes
Lattice and Batch and, where a program keeps its fields in page-locked memory,
the C ABI calls under them (include/sfh.h).  Sizes, masses, step sizes and
tolerances are those of the repository's own benchmark configurations: plain
FP64 HMC at 4^4, the 16^4 operator and solver grid, the 32^3 x 64 solve, the
uneven batch drawn from {8^4, 12^4, 16^4, 16^3 x 32}, and 24^4 HMC with a
Hasenbusch pair on stout links; draw() spreads over the ranges between them,
uneven extents included.

Fields are in the reference layouts: links, momenta and forces
double[V][4][3][3][2], spinors double[V][3][2], site
((x Ly + y) Lz + z) Lt + t.
"""
import ctypes
import math
import random

import torch

import staggered_fermions_hmc_b200 as sfh

TOL = 1e-10  # relative residual of the solves, as the benchmark configurations
MD_TOL = 1e-12  # leapfrog's own default: reversible molecular dynamics
MAXIT = 20000
BETA, C11, C12 = 4.2, 5.0 / 3.0, -1.0 / 12.0
HEX_ALPHAS = (0.95, 0.76, 0.38)
BATCH_LATTICES = "8x8x8x8,12x12x12x12,16x16x16x16,16x16x16x32"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # D D^dag of one vector on the smallest lattice: a call's fixed cost
        dict(name="apply_4x4", kind="apply", dims="4x4x4x4", mass=0.1, eps=0.3),
        # the plain FP64 HMC configuration, one whole update of 10 leapfrog steps
        dict(name="trajectory_4x4_f64", kind="trajectory", dims="4x4x4x4", mass=0.1, eps=0.3, dt=0.1, steps=10,
             precision="f64", heavy=0.0, rho=0.0, levels=0),
        # molecular dynamics of a production run on thin links: mixed solves,
        # both forces, link updates, from given momenta and pseudofermion
        dict(name="leapfrog_12x24_f32", kind="leapfrog", dims="12x12x12x24", mass=0.1, eps=0.3, dt=0.02, steps=6,
             precision="f32"),
        # three steps of the 24^4 configuration: Hasenbusch pair, 4 stout levels
        dict(name="trajectory_24x4_stout_f32", kind="trajectory", dims="24x24x24x24", mass=0.02, eps=0.3, dt=0.01,
             steps=3, precision="f32", heavy=0.2, rho=0.125, levels=4),
        # one propagator in plain FP64 on a small lattice (the reference's own solve)
        dict(name="solve_8x16_f64", kind="solve", dims="8x8x8x16", mass=0.1, eps=1.0, precision="f64"),
        # one propagator in mixed precision on rough links
        dict(name="solve_16x4_f16", kind="solve", dims="16x16x16x16", mass=0.05, eps=1.0, precision="f16"),
        # one propagator on the largest lattice
        dict(name="solve_32x64_f16", kind="solve", dims="32x32x32x64", mass=0.1, eps=1.0, precision="f16"),
        # a third of the uneven batch: independent lattices, masses, 1-8 sources each
        dict(name="batch_f16", kind="batch", lattices=BATCH_LATTICES, systems=20, spec=7, precision="f16"),
        # a few small, ragged lattices solved together in FP64
        dict(name="batch_small_f64", kind="batch", lattices="4x6x10x14,6x6x6x10,8x4x6x18,10x10x10x10", systems=6,
             spec=3, precision="f64"),
        # pure-gauge updates with a measurement: sweeps, plaquette, action, Polyakov loops
        dict(name="heatbath_16x4", kind="heatbath", dims="16x16x16x16", eps=0.3, beta=4.2, sweeps=5),
        # the smearing of a stored configuration, as Apply_4HEX_smearing
        dict(name="hex4_16x32", kind="smear", dims="16x16x16x32", eps=0.3, hexes=4, stouts=0, rho=0.0),
        # the full force on given X and Y (a caller with its own integrator)
        dict(name="force_16x4", kind="force", dims="16x16x16x16", mass=0.1, eps=0.3),
    ]


def _draw_dims(rng, low, high, step=2):
    """Four extents, multiples of step, their product spread over [low, high]
    in its logarithm."""
    want = math.exp(rng.uniform(math.log(low), math.log(high)))
    while True:
        d = [step * max(1, round(want ** 0.25 * math.exp(rng.gauss(0.0, 0.3)) / step)) for _ in range(4)]
        if min(d) >= 4 and low <= math.prod(d) <= high:
            return "x".join(map(str, d))


def draw(rng):
    kind = rng.choice(["apply", "trajectory", "trajectory", "leapfrog", "solve", "solve", "solve", "batch", "batch",
                       "heatbath", "smear", "force"])
    mass, eps = round(math.exp(rng.uniform(math.log(0.05), math.log(0.2))), 4), round(rng.uniform(0.3, 1.0), 3)
    if kind in ("apply", "force"):
        return dict(kind=kind, dims=_draw_dims(rng, 256, 16 ** 4), mass=mass, eps=eps)
    if kind in ("trajectory", "leapfrog"):
        case = dict(kind=kind, dims=_draw_dims(rng, 256, 16 ** 4), mass=mass, eps=round(rng.uniform(0.2, 0.4), 3),
                    dt=round(rng.uniform(0.01, 0.03), 4), steps=rng.randint(2, 6),
                    precision=rng.choice(["f64", "f32", "f16"]))
        if kind == "trajectory":
            stout, pair = rng.random() < 0.5, rng.random() < 0.5
            case.update(heavy=0.3 if pair else 0.0, rho=0.125 if stout else 0.0,
                        levels=rng.randint(1, 4) if stout else 0)
        return case
    if kind == "solve":
        return dict(kind=kind, dims=_draw_dims(rng, 256, 24 ** 3 * 48), mass=mass, eps=eps,
                    precision=rng.choice(["f64", "f32", "f32_18", "f16", "bf16"]))
    if kind == "batch":
        precision = rng.choice(["f64", "f32", "f16", "f16"])
        lattices = ",".join(_draw_dims(rng, 256, 12 ** 4 if precision == "f64" else 16 ** 4) for _ in range(3))
        return dict(kind=kind, lattices=lattices, systems=rng.randint(2, 10), spec=rng.randrange(1 << 20),
                    precision=precision)
    if kind == "heatbath":
        return dict(kind=kind, dims=_draw_dims(rng, 256, 16 ** 4, step=4), eps=round(rng.uniform(0.2, 0.6), 3),
                    beta=round(rng.uniform(2.0, 6.0), 3), sweeps=rng.randint(1, 8))
    hexes = rng.randint(0, 4)
    return dict(kind="smear", dims=_draw_dims(rng, 256, 16 ** 3 * 32), eps=round(rng.uniform(0.2, 0.4), 3),
                hexes=hexes, stouts=rng.randint(1, 6) if hexes < 2 else 0, rho=round(rng.uniform(0.05, 0.125), 4))


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
def _dims(text):
    return tuple(int(v) for v in text.split("x"))


def _volume(text):
    return math.prod(_dims(text))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed % (1 << 62))


def _hermitian(gen, n, scale):
    """n traceless Hermitian 3x3 matrices with N(0, scale^2) entries."""
    z = scale * torch.randn(n, 9, generator=gen, device="cuda", dtype=torch.float64)
    h = torch.zeros(n, 3, 3, device="cuda", dtype=torch.complex128)
    for k, (a, b) in enumerate(((0, 1), (0, 2), (1, 2))):
        h[:, a, b] = torch.complex(z[:, 3 + 2 * k], z[:, 4 + 2 * k])
        h[:, b, a] = h[:, a, b].conj()
    diag = z[:, :3] - z[:, :3].mean(1, keepdim=True)
    for k in range(3):
        h[:, k, k] = diag[:, k]
    return h


def _expm(h, factor):
    """exp(i factor h), a million matrices at a time (bounds the work space)."""
    out = torch.empty_like(h)
    for k in range(0, h.shape[0], 1 << 20):
        out[k:k + (1 << 20)] = torch.linalg.matrix_exp(1j * factor * h[k:k + (1 << 20)])
    return out


def _links(gen, dims, eps):
    """U = exp(i eps H) on every link: the seeded hot start."""
    return _expm(_hermitian(gen, 4 * math.prod(dims), 1.0), eps).view(*dims, 4, 3, 3)


def _momenta(gen, dims):
    """P = sum_a p_a lambda_a / 2 with p_a ~ N(0, 1)."""
    n = 4 * math.prod(dims)
    p = 0.5 * torch.randn(n, 8, generator=gen, device="cuda", dtype=torch.float64)
    h = torch.zeros(n, 3, 3, device="cuda", dtype=torch.complex128)
    for k, (a, b) in enumerate(((0, 1), (0, 2), (1, 2))):
        h[:, a, b] = torch.complex(p[:, 2 * k], -p[:, 2 * k + 1])
        h[:, b, a] = h[:, a, b].conj()
    l8 = p[:, 7] / math.sqrt(3.0)
    h[:, 0, 0], h[:, 1, 1], h[:, 2, 2] = (p[:, 6] + l8).to(h.dtype), (l8 - p[:, 6]).to(h.dtype), (-2 * l8).to(h.dtype)
    return h.view(*dims, 4, 3, 3)


def _source(gen, dims, n=1):
    """n complex Gaussian vectors of variance 1/2 per real part."""
    z = torch.randn(n, *dims, 3, 2, generator=gen, device="cuda", dtype=torch.float64) * math.sqrt(0.5)
    return torch.view_as_complex(z)


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True)


def _host(field):
    """A device field as a flat page-locked float64 array in the reference layout."""
    flat = torch.view_as_real(field.contiguous()).reshape(-1)
    out = _pinned(flat.numel())
    out.copy_(flat)
    return out.numpy()


def _batch_spec(case):
    """[(dims, mass, nrhs, eps)] of an uneven batch."""
    rng = random.Random(case["spec"])
    names = case["lattices"].split(",")
    return [(_dims(rng.choice(names)), rng.choice([0.05, 0.1, 0.2]), rng.randint(1, 8), rng.choice([0.3, 1.0]))
            for _ in range(case["systems"])]


def _inputs(case, seed):
    """The fields of a case on the GPU."""
    gen = _generator(seed)
    if case["kind"] == "batch":
        return [(_links(gen, dims, eps), _source(gen, dims, nrhs)) for dims, _, nrhs, eps in _batch_spec(case)]
    dims = _dims(case["dims"])
    f = {"U": _links(gen, dims, case["eps"])}
    if case["kind"] in ("apply", "solve"):
        f["psi"] = _source(gen, dims)[0]
    elif case["kind"] == "leapfrog":
        f["P"] = _momenta(gen, dims)
        f["phi"] = _Staggered(f["U"], case["mass"]).dirac(_source(gen, dims)[0])
    elif case["kind"] == "force":
        f["X"], f["Y"] = _source(gen, dims, 2)
    return f


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def _ptr(array):
    return array.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def prepare(case, seed):
    kind = case["kind"]
    fields = _inputs(case, seed)
    if kind == "batch":
        spec = _batch_spec(case)
        batch = sfh.Batch([(dims, mass, nrhs) for dims, mass, nrhs, _ in spec], precision=case["precision"])
        out = _pinned(sum(6 * math.prod(dims) * nrhs for dims, _, nrhs, _ in spec)).numpy()
        slots, at = [], 0
        for k, ((dims, _, nrhs, _), (U, phi)) in enumerate(zip(spec, fields)):
            batch.set_gauge(k, _host(U))
            for j in range(nrhs):
                batch.set_rhs(k, j, _host(phi[j]))
                slots.append((k, j, out[at:at + 6 * math.prod(dims)]))
                at += 6 * math.prod(dims)
        return dict(kind=kind, case=case, batch=batch, out=out, slots=slots)
    dims = _dims(case["dims"])
    lat = sfh.Lattice(dims, case.get("mass", 0.1), beta=case.get("beta", BETA))
    state = dict(kind=kind, case=case, lat=lat, seed=seed)
    host = {k: _host(v) for k, v in fields.items()}
    if kind in ("apply", "solve", "force"):
        lat.upload_gauge(host["U"])  # these read the links they were given
    state.update(host)
    if kind in ("trajectory", "leapfrog", "heatbath", "smear", "force"):
        state["links"] = _pinned(72 * lat.V).numpy()
    if kind == "leapfrog":
        state["momenta"] = _pinned(72 * lat.V).numpy()
    if kind == "trajectory":
        if case["heavy"] > 0.0:
            lat.set_hasenbusch(case["heavy"])
        if case["levels"] > 0:
            lat.set_fermion_smearing(case["rho"], case["levels"])
    return state


def _check(status):
    if status != sfh.SFH_OK:
        raise sfh.SfhError(status, "call failed")


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "batch":
        state["batch"].solve(tol=TOL, max_iter=MAXIT)
        for k, j, view in state["slots"]:
            state["batch"].solution(k, j, out=view)
        return state["out"]
    lat = state["lat"]
    if kind == "apply":
        return lat.apply_DDdagger(state["psi"])
    if kind == "solve":
        return lat.solve_CG_DDdagger(state["psi"], tol=TOL, max_iter=MAXIT, precision=case["precision"])
    if kind == "force":
        _check(lat.lib.sfh_full_force(lat.h, _ptr(state["X"]), _ptr(state["Y"]), _ptr(state["links"])))
        return state["links"]
    # the others start from a stored configuration and leave an updated one
    lat.upload_gauge(state["U"])
    out = {}
    if kind == "trajectory":
        info = lat.hmc_trajectory(case["dt"], case["steps"], state["seed"], tol=TOL, max_iter=MAXIT,
                                  precision=case["precision"])
        out = {"H": torch.tensor(info["H_initial"] + info["H_final"], dtype=torch.float64),
               "plaquette": info["plaquette"]}
    elif kind == "leapfrog":
        lat.upload_momenta(state["P"])
        out["X"], _ = lat.leapfrog(state["phi"], case["dt"], case["steps"], tol=MD_TOL, max_iter=MAXIT,
                                   precision=case["precision"])
        _check(lat.lib.sfh_download_momenta(lat.h, _ptr(state["momenta"])))
        out["momenta"] = state["momenta"]
    elif kind == "heatbath":
        out["plaquette"], out["action"] = lat.heatbath_update(case["sweeps"], seed=state["seed"] % (1 << 31))
        out["polyakov"] = lat.precompute_polyakov_grid()
    else:
        if case["stouts"]:
            lat.smear_stout(case["rho"], case["stouts"])
        if case["hexes"]:
            lat.Apply_HEX_smearing(HEX_ALPHAS, passes=case["hexes"])
        out["plaquette"] = lat.compute_avg_plaq()
    _check(lat.lib.sfh_download_gauge(lat.h, _ptr(state["links"])))
    out["links"] = state["links"]
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
MATRIX = 198  # flops of a 3x3 complex product
CACHE = 126e6  # fields that fit in L2 need not be read from memory again
LINK_BYTES = {"f64": 576, "f32": 192, "f32_18": 288, "f16": 96, "bf16": 96}  # four links
SPINOR_BYTES = {"f64": 48, "f32": 24, "f32_18": 24, "f16": 16, "bf16": 16}


def _iterations(mass, eps):
    """CG iterations to 1e-10 on exp(i eps H) links (measured, smoothed)."""
    return 32.5 / mass if eps > 0.6 else 133.0 * (0.2 / mass) ** 0.88


def _solve_work(V, nrhs, mass, eps, precision):
    """Links and sources in, solutions out, and per iteration two hops (links
    and vectors) and the vector updates where the fields exceed the L2."""
    s, lb = SPINOR_BYTES[precision], LINK_BYTES[precision]
    its = _iterations(mass, eps)
    once = V * (576 + 96 * nrhs)
    again = V * (2 * lb + nrhs * 11 * s) if V * (lb + 4 * nrhs * s) > CACHE else 0
    return once + its * again, its * V * nrhs * (2 * 570 + 100)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [_solve_work(math.prod(d), n, m, e, case["precision"]) for d, m, n, e in _batch_spec(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    V = _volume(case["dims"])
    # gauge force per link: 12 products for the two-sided staples of the
    # adjacent links, 30 for the plaquette and rectangle sums, one for U V
    force = V * 4 * 43 * MATRIX
    if kind == "apply":
        return {"bytes": V * (576 + 96), "flops": V * 2 * 570}
    if kind == "solve":
        b, f = _solve_work(V, 1, case["mass"], case["eps"], case["precision"])
        return {"bytes": b, "flops": f}
    if kind == "force":
        return {"bytes": V * (2 * 576 + 96), "flops": force + V * 4 * 3 * MATRIX}
    if kind == "heatbath":
        n = case["sweeps"]
        return {"bytes": V * 2 * 576 * n, "flops": n * V * 4 * (70 + 6) * MATRIX}
    stout = V * 4 * 18 * MATRIX  # six staples, the exponential, the product
    if kind == "smear":
        return {"bytes": V * 2 * 576, "flops": case["stouts"] * stout + case["hexes"] * V * 4 * 99 * MATRIX}
    solves = case["steps"] + (2 if kind == "trajectory" else 1)
    b, f = _solve_work(V, 1, case["mass"], case["eps"], case["precision"])
    levels = case.get("levels", 0)
    if case.get("heavy", 0.0) > 0.0:
        b2, f2 = _solve_work(V, 1, case["heavy"], case["eps"], case["precision"])
        b, f = b + b2, f + f2
    step = V * 576 * (6 + 12 * levels)
    return {"bytes": solves * (b + step), "flops": solves * (f + force + 4 * levels * stout + V * 4 * 10 * MATRIX)}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _shift(f, mu, n):
    """f(x + n mu) on a field whose leading four axes are the lattice."""
    return torch.roll(f, -n, mu)


def _adj(m):
    return m.conj().transpose(-1, -2)


class _Staggered:
    """D = m + K on links U: K psi(x) = sum_mu eta_mu / 2 (U_mu(x) psi(x + mu)
    - U_mu(x - mu)^dag psi(x - mu)), antiperiodic in t."""

    def __init__(self, U, mass):
        dims = U.shape[:4]
        self.mass = mass
        x = torch.meshgrid(*(torch.arange(n, device=U.device) for n in dims), indexing="ij")
        self.eta, self.fwd, self.bwd = [], [], []
        for mu in range(4):
            eta = (1 - 2 * (sum(x[:mu], torch.zeros_like(x[0])) % 2)).to(torch.float64)
            if mu == 3:
                wrap = torch.where(x[3] == dims[3] - 1, -1.0, 1.0).to(torch.float64)
            else:
                wrap = torch.ones_like(eta)
            self.eta.append(eta * wrap)  # of the forward hop; the backward one takes the neighbour's
            half = 0.5 * (eta * wrap)[..., None, None]
            self.fwd.append(half * U[..., mu, :, :])
            self.bwd.append(_shift(_adj(half * U[..., mu, :, :]), mu, -1))

    def hop(self, psi):
        """K of one vector or of a stack of them (a leading axis)."""
        lead = psi.dim() - 5
        out = torch.zeros_like(psi)
        for mu in range(4):
            up, dn = _shift(psi, mu + lead, 1), _shift(psi, mu + lead, -1)
            for c in range(3):
                out += self.fwd[mu][..., c] * up[..., c, None] - self.bwd[mu][..., c] * dn[..., c, None]
        return out

    def dirac(self, psi):
        return self.mass * psi + self.hop(psi)

    def dagger(self, psi):
        return self.mass * psi - self.hop(psi)

    def normal(self, psi):
        return self.mass ** 2 * psi - self.hop(self.hop(psi))

    def solve(self, b, tol=1e-14):
        """(D D^dag)^-1 b for a stack of vectors by conjugate gradients."""
        axes = tuple(range(1, b.dim()))

        def dot(u, v):
            return (torch.view_as_real(u) * torch.view_as_real(v)).flatten(1).sum(1)

        def wide(s):
            return s.view(-1, *[1] * len(axes))

        x, r = torch.zeros_like(b), b.clone()
        p, rr = r.clone(), dot(r, r)
        stop = tol * tol * rr
        for it in range(MAXIT):
            v = self.normal(p)
            alpha = rr / dot(p, v)
            x += wide(alpha) * p
            r -= wide(alpha) * v
            new = dot(r, r)
            p = r + wide(new / rr) * p
            rr = new
            if it % 16 == 15 and bool((rr <= stop).all()):
                break
        return x


def _path(U, mu, steps):
    """Product of links along signed steps (+-(nu + 1)) from x + mu."""
    at, out = [0, 0, 0, 0], None
    at[mu] = 1

    def link(nu):
        f = U[..., nu, :, :]
        shifts = [(-s, d) for d, s in enumerate(at) if s]
        return torch.roll(f, [s for s, _ in shifts], [d for _, d in shifts]) if shifts else f

    for s in steps:
        nu = abs(s) - 1
        if s > 0:
            m = link(nu)
            at[nu] += 1
        else:
            at[nu] -= 1
            m = _adj(link(nu))
        out = m if out is None else out @ m
    return out


def _gauge_force(U, beta):
    out = []
    for mu in range(4):
        M, V = mu + 1, 0
        for nu in range(4):
            if nu == mu:
                continue
            for s in (1, -1):
                N = s * (nu + 1)
                V = V + C11 * _path(U, mu, (N, -M, -N))
                for steps in ((N, N, -M, -N, -N), (M, N, -M, -M, -N), (N, -M, -M, -N, M)):
                    V = V + C12 * _path(U, mu, steps)
        out.append(U[..., mu, :, :] @ V)
    Q = torch.stack(out, -3)
    return _traceless(-1j * (beta / 12.0) * (Q - _adj(Q)))


def _traceless(m):
    t = torch.diagonal(m, dim1=-2, dim2=-1).mean(-1)
    return m - t[..., None, None] * torch.eye(3, device=m.device, dtype=m.dtype)


def _outer(a, b):
    return a[..., :, None] * b.conj()[..., None, :]


def _fermion_force(D, U, X, Y):
    out = []
    for mu in range(4):
        u = U[..., mu, :, :]
        Xu, Yu = _shift(X, mu, 1), _shift(Y, mu, 1)
        S = _outer((u @ Yu[..., None])[..., 0], X) + _outer(Y, Xu) @ _adj(u)
        out.append(-0.25j * D.eta[mu][..., None, None] * (S - _adj(S)))
    return _traceless(torch.stack(out, -3))


def _leapfrog(U, P, phi, mass, dt, steps):
    def kick(h):
        D = _Staggered(U, mass)
        X = D.solve(phi[None])[0]
        return P - h * (_gauge_force(U, BETA) + _fermion_force(D, U, X, D.dagger(X))), X

    P, X = kick(0.5 * dt)
    for n in range(steps):
        U = _expm(P.reshape(-1, 3, 3), dt).view_as(U) @ U
        P, X = kick(dt if n < steps - 1 else 0.5 * dt)
    return U, P, X


def _staple(side, middle, mu, nu):
    """The two-sided staple from x to x + mu through nu."""
    up = side @ _shift(middle, nu, 1) @ _adj(_shift(side, mu, 1))
    return up + _shift(_adj(side) @ middle @ _shift(side, mu, 1), nu, -1)


def _smeared(G, u, c):
    om = G @ _adj(u)
    h = _traceless(-0.5j * (om - _adj(om)))  # exp(c A) = exp(i c (-i A))
    return _expm(h.reshape(-1, 3, 3), c).view_as(u) @ u


def _stout(U, rho):
    return torch.stack([_smeared(sum(_staple(U[..., n, :, :], U[..., m, :, :], m, n) for n in range(4) if n != m),
                                 U[..., m, :, :], rho) for m in range(4)], -3)


def _hex(U):
    a1, a2, a3 = (0.5 * a for a in HEX_ALPHAS)
    u = [U[..., m, :, :] for m in range(4)]
    V1, V2 = {}, {}
    for m in range(4):
        for r in range(4):
            if r != m:
                V1[m, r] = _smeared(_staple(u[r], u[m], m, r), u[m], a3)
    for m in range(4):
        for n in range(4):
            if n != m:
                rest = [s for s in range(4) if s not in (m, n)]
                G = sum(_staple(V1[s, 6 - m - n - s], V1[m, 6 - m - n - s], m, s) for s in rest)
                V2[m, n] = _smeared(G, u[m], a2)
    return torch.stack([_smeared(sum(_staple(V2[n, m], V2[m, n], m, n) for n in range(4) if n != m), u[m], a1)
                        for m in range(4)], -3)


def _plaquette(U):
    """Six times the average plaquette: 6 on a cold field."""
    total = 0.0
    for m in range(4):
        for n in range(m):
            um, un = U[..., m, :, :], U[..., n, :, :]
            p = um @ _shift(un, m, 1) @ _adj(_shift(um, n, 1)) @ _adj(un)
            total += torch.diagonal(p, dim1=-2, dim2=-1).real.sum().item() / 3.0
    return total / math.prod(U.shape[:4])


def _flat(field):
    return torch.view_as_real(field.contiguous()).reshape(-1)


# seconds of _Staggered.solve per iteration: launches, and per site and vector
SOLVE_SECONDS = (1e-3, 3.5e-9)


def _seconds(V, nrhs, mass, eps):
    return 1.3 * _iterations(mass, eps) * (SOLVE_SECONDS[0] + SOLVE_SECONDS[1] * V * nrhs)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("trajectory", "heatbath"):
        return None  # their random fields are drawn by the library
    if kind == "batch":
        spec = _batch_spec(case)
        if sum(_seconds(math.prod(d), n, m, e) for d, m, n, e in spec) > 20.0:
            return None
        return torch.cat([_flat(_Staggered(U, mass).solve(phi))
                          for (_, mass, _, _), (U, phi) in zip(spec, _inputs(case, seed))])
    if kind in ("solve", "leapfrog"):
        n = case["steps"] + 1 if kind == "leapfrog" else 1
        if n * _seconds(_volume(case["dims"]), 1, case["mass"], case["eps"]) > 20.0:
            return None
    f = _inputs(case, seed)
    if kind == "apply":
        return _flat(_Staggered(f["U"], case["mass"]).normal(f["psi"]))
    if kind == "solve":
        return _flat(_Staggered(f["U"], case["mass"]).solve(f["psi"][None])[0])
    if kind == "force":
        D = _Staggered(f["U"], case["mass"])
        return _flat(_gauge_force(f["U"], BETA) + _fermion_force(D, f["U"], f["X"], f["Y"]))
    if kind == "leapfrog":
        U, P, X = _leapfrog(f["U"], f["P"], f["phi"], case["mass"], case["dt"], case["steps"])
        return {"X": _flat(X), "momenta": _flat(P), "links": _flat(U)}
    U = f["U"]
    for _ in range(case["stouts"]):
        U = _stout(U, case["rho"])
    for _ in range(case["hexes"]):
        U = _hex(U)
    return {"plaquette": _plaquette(U), "links": _flat(U)}
