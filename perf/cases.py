"""What a user of the sphere finite-element library has it do, as measurable cases.

``listed()`` are twelve calls of the public Python API, over the mesh levels 3 to 7 that the serving trace and the
benchmark use; ``draw(rng)`` gives more calls of the same kinds and ranges.  ``prepare`` builds the inputs on the GPU
(spherical-harmonic fields, as every workload of this repository uses them) and takes the operator set and the time
stepper of the mesh, which a program creates once and keeps; ``run`` is one call; ``exact`` is the same result by plain
torch in 64 bits, from the assembled matrices of the mesh.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from mke_gb300 import phelm

# the barotropic and baroclinic configurations of the benchmark
BV = dict(tau=1e-3, sigma=1.6e-2, mu=8e-5, k1=1.0, k2=1.0, theta=0.5, picard_iters=3)
BC = dict(tau=1e-3, sigma=0.05, mu=6.77e-5, sigma1=0.05, mu1=6.77e-5, alpha=0.1 ** 0.5, picard_iters=3,
          picard_tol=1e-8)
TOL = 1e-12   # the library's default solve tolerance


def listed():
    def case(name, kind, level, mixed, members=1, steps=1):
        return dict(name=name, kind=kind, level=level, mixed=mixed, members=members, steps=steps)

    return [
        # one Poisson solve on the smallest mesh in use (642 points): launch and barrier latency
        case("solve_l3_fp64", "solve", 3, False),
        # one Poisson solve on the largest mesh of the serving trace (163,842 points)
        case("solve_l7_mixed", "solve", 7, True),
        # the Poisson solves that a serving turn finds waiting on one mesh, an odd number of them
        case("solve_batch_l5x37_mixed", "solve", 5, True, members=37),
        # the vorticity of a stream function: one Laplacian with its mass solve
        case("laplacian_l6_fp64", "laplacian", 6, False),
        # one Jacobian J(u, v): eight derivatives, eight mass solves
        case("jacobian_l6_fp64", "jacobian", 6, False),
        # the headline: a barotropic trajectory at level 6, stepped in place as captured steps
        case("run_l6_mixed", "run", 6, True, steps=4),
        # the same model in double, one step per call (a program that looks at each state)
        case("step_l6_fp64", "step", 6, False),
        # a served request: a ten-step integration on a small mesh
        case("run_l4_mixed", "run", 4, True, steps=10),
        # the batched ensemble: 256 perturbed members at level 5
        case("ensemble_l5x256_mixed", "step", 5, True, members=256),
        # the adjoint of the linearised step (sensitivity studies: the backward direction)
        case("adjoint_l6_fp64", "adjoint", 6, False),
        # the two-layer baroclinic model
        case("baroclin_l6_mixed", "baroclin", 6, True),
        # the bare FP32 operator apply on an interleaved multi-vector, larger than the L2
        case("mult32_l7x128", "mult32", 7, True, members=128),
    ]


def draw(rng):
    """One more case: each kind over the levels and member counts it is used at, none dearer than the listed ones."""
    kind = rng.choice(["solve", "solve", "batch", "batch", "laplacian", "jacobian", "run", "step", "ensemble",
                       "ensemble", "adjoint", "baroclin", "mult32"])
    mixed, level, members, steps = rng.random() < 0.5, rng.randint(3, 7), 1, 1

    def spread(lo, hi):   # whole numbers, even over their logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "batch":
        kind, level = "solve", rng.randint(3, 6)
        members = spread(2, {3: 200, 4: 200, 5: 120, 6: 40}[level])
    elif kind == "ensemble":
        kind, level, mixed = "step", rng.randint(3, 6), rng.random() < 0.75
        most = {3: 256, 4: 256, 5: 256, 6: 32}[level]
        members = spread(2, most if mixed else most // 8)
    elif kind == "run":
        level, steps = rng.randint(3, 6), rng.randint(2, 4)
    elif kind in ("step", "adjoint", "baroclin"):
        level = rng.randint(3, 6)
    elif kind == "mult32":
        level, mixed, members = rng.randint(5, 7), True, 4 * 2 ** rng.randint(0, 5)
    return dict(kind=kind, level=level, mixed=mixed, members=members, steps=steps)


# ------------------------------------------------------------------ what a program keeps: mesh, operators, steppers

@functools.lru_cache(maxsize=None)
def _mesh(level):
    return phelm.Mesh.sphere(level)


@functools.lru_cache(maxsize=None)
def _ops(level, mixed):
    return phelm.Operators(_mesh(level), phelm.PHG_MIXED if mixed else phelm.PHG_FP64, tol=TOL)


@functools.lru_cache(maxsize=None)
def _barvortex(level, mixed):
    lat, _ = _mesh(level).latlon()
    return phelm.BarVortex(_ops(level, mixed), coriolis=np.sin(lat), **BV)


@functools.lru_cache(maxsize=None)
def _baroclin(level, mixed):
    lat, _ = _mesh(level).latlon()
    return phelm.Baroclin(_ops(level, mixed), coriolis=np.sin(lat), **BC)


@functools.lru_cache(maxsize=None)
def _stream():
    return torch.cuda.Stream()   # the program's compute stream


@functools.lru_cache(maxsize=None)
def _harmonics(level, lmax):
    """Real orthonormal spherical harmonics of degrees 1..lmax at the points (modes x V), and each mode's degree."""
    lat, lon = (torch.tensor(a, device="cuda") for a in _mesh(level).latlon())
    x, c = torch.sin(lat), torch.cos(lat)
    rows, degree = [], []
    p_mm = torch.full_like(x, 1.0 / math.sqrt(4.0 * math.pi))
    for m in range(lmax + 1):
        if m:
            p_mm = -math.sqrt((2.0 * m + 1.0) / (2.0 * m)) * c * p_mm
        before, p = torch.zeros_like(x), p_mm
        for l in range(m, lmax + 1):
            if l > m:
                a = math.sqrt((4.0 * l * l - 1.0) / (l * l - m * m))
                b = math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1.0) ** 2 - 1.0)) if l > m + 1 else 0.0
                before, p = p, a * (x * p - b * before)
            if l == 0:
                continue
            if m == 0:
                rows.append(p)
                degree.append(l)
            else:
                rows += [math.sqrt(2.0) * p * torch.cos(m * lon), math.sqrt(2.0) * p * torch.sin(m * lon)]
                degree += [l, l]
    return torch.stack(rows), torch.tensor(degree, dtype=torch.float64, device="cuda")


def _random_field(level, lmax, members, seed, amplitude):
    """members x V: sum of c Y, c Gaussian with norm `amplitude`; and the stream function whose Laplacian it is."""
    Y, l = _harmonics(level, lmax)
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.randn(members, Y.shape[0], generator=g, device="cuda", dtype=torch.float64)
    c *= amplitude / c.norm(dim=1, keepdim=True)
    return c @ Y, (-c / (l * (l + 1.0))) @ Y


def _wave_state(level, members, seed):
    """Stream functions of a wavenumber-4 Rossby-Haurwitz wave (amplitude 0.1) with noise (degree <= 16, 1e-3)."""
    lat, lon = (torch.tensor(a, device="cuda") for a in _mesh(level).latlon())
    wave = 0.1 * torch.cos(lat) ** 4 * torch.sin(lat) * torch.cos(4.0 * lon) / -30.0
    return (wave + _random_field(level, 16, members, seed, 1e-3)[1]).contiguous()


def _inputs(case, seed):
    kind, level, members = case["kind"], case["level"], case["members"]
    if kind == "solve":   # right-hand sides of degree <= 10, a value at the pole
        F = _random_field(level, 10, members, seed, 1.0)[0]
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        bnd = 0.1 * torch.randn(members, _mesh(level).outer_size, generator=g, device="cuda", dtype=torch.float64)
        return dict(F=F, bnd=bnd)
    if kind == "mult32":
        g = torch.Generator(device="cuda").manual_seed(seed)
        return dict(x=torch.randn(_mesh(level).inner_size, members, generator=g, device="cuda"))
    if kind == "laplacian":
        return dict(u=_wave_state(level, 1, seed)[0])
    if kind == "jacobian":
        return dict(u=_random_field(level, 12, 1, seed, 0.05)[1][0], v=_random_field(level, 12, 1, seed + 1, 0.05)[0][0])
    if kind == "adjoint":   # a perturbation, and the state that the step is linearised around
        return dict(u=_random_field(level, 12, 1, seed, 0.05)[1][0], z=_wave_state(level, 1, seed + 1)[0])
    if kind == "baroclin":
        return dict(u1=_random_field(level, 12, 1, seed, 0.05)[1][0], u2=_random_field(level, 12, 1, seed + 1, 0.05)[1][0])
    return dict(u=_wave_state(level, members, seed))


def prepare(case, seed):
    kind, level, mixed = case["kind"], case["level"], case["mixed"]
    s = dict(case=case, stream=_stream(), **_inputs(case, seed))
    m = _mesh(level)
    if kind in ("run", "step", "adjoint"):
        s["model"] = _barvortex(level, mixed)
    elif kind == "baroclin":
        s["model"] = _baroclin(level, mixed)
    else:
        s["ops"] = _ops(level, mixed)
    if kind == "mult32":
        s["out"] = torch.empty_like(s["x"])
    elif kind == "baroclin":
        s["out"] = torch.empty(2, m.size, dtype=torch.float64, device="cuda")
    elif kind == "solve":
        s["out"] = torch.empty_like(s["F"])
    else:
        s["out"] = torch.empty_like(s["u"])
    torch.cuda.synchronize()   # the inputs are complete before the compute stream reads them
    return s


def run(s):
    case, st, out = s["case"], s["stream"], s["out"]
    kind = case["kind"]
    if kind == "solve":
        lap = phelm.SphereLaplace(s["ops"])
        if case["members"] == 1:
            lap.solve(s["F"], s["bnd"], out=out, stream=st)
        else:
            lap.solve_batch(s["F"], s["bnd"], out=out, stream=st)
    elif kind == "laplacian":
        phelm.SphereLaplace(s["ops"]).calc1(s["u"], out=out, stream=st)
    elif kind == "jacobian":
        phelm.SphereJacobian(s["ops"]).calc1(s["u"], s["v"], out=out, stream=st)
    elif kind == "run":
        with torch.cuda.stream(st):
            out.copy_(s["u"])   # a new trajectory starts
        s["model"].run(out, case["steps"], stream=st)
    elif kind == "step":
        s["model"].calc_batch(s["u"], out=out, stream=st)
    elif kind == "adjoint":
        s["model"].calc_LT(s["u"], s["z"], out=out, stream=st)
    elif kind == "baroclin":
        s["model"].calc(s["u1"], s["u2"], out1=out[0], out2=out[1], stream=st)
    else:
        s["ops"].mult32("lapl", s["x"], out, stream=st)
    return out


def work(case):
    """Inputs, outputs and the matrices of the path once each; a multiply and an add per nonzero that the path applies
    at least once (a solve applies its matrix at least once per right-hand side)."""
    kind, members, steps = case["kind"], case["members"], case["steps"]
    n = 10 * 4 ** case["level"] + 2
    nnz = 7 * n
    if kind == "mult32":
        return dict(bytes=8 * nnz + 8 * n * members, flops=2 * nnz * members)
    # (matrices of 8-byte values on one 4-byte pattern, fields in and out, matrix applications of one pass)
    mats, fields, applies = {
        "solve": (2, 2, 2),
        "laplacian": (2, 2, 2),
        "jacobian": (5, 3, 16),
        "adjoint": (8, 3, 2 * 5 + 3 * 16 + 4),
        "baroclin": (12, 4, 2 * 4 + 3 * (5 * 16 + 2 + 9)),
        "run": (8, 2, steps * (4 + 3 * (16 + 4))),
        "step": (8, 2, steps * (4 + 3 * (16 + 4))),
    }[kind]
    return dict(bytes=nnz * (4 + 8 * mats) + 8 * n * fields * members, flops=2 * nnz * applies * members)


# ---------------------------------------------------------------- the same results by plain torch in 64 bits

class _Discrete:
    """The assembled matrices of one mesh (the data of the problem) as torch tensors; vectors are columns."""

    def __init__(self, level):
        m = _mesh(level)
        maps = m.maps()
        self.V, self.rs, self.os = m.size, m.inner_size, m.outer_size
        self.inner, self.outer = (torch.tensor(maps[k], device="cuda").long() for k in ("inner", "outer"))
        self.m, self.mats = m, {}
        lat, _ = m.latlon()
        self.coriolis = torch.sin(torch.tensor(lat, device="cuda"))[:, None]

    def mat(self, name):
        if name not in self.mats:
            ptr, col, val = self.m.csr(name)
            rows = len(ptr) - 1
            cols = self.os if "b" in name or name.startswith("bnd") else self.V if name == "norm" else self.rs
            self.mats[name] = torch.sparse_csr_tensor(torch.tensor(ptr).long(), torch.tensor(col).long(),
                                                      torch.tensor(val), size=(rows, cols)).cuda()
        return self.mats[name]

    def diag(self, name):
        a = self.mat(name).to_sparse_coo().coalesce()
        i, j = a.indices()
        d = torch.zeros(self.rs, dtype=torch.float64, device="cuda")
        d[i[i == j]] = a.values()[i == j]
        return d[:, None]

    def full(self, x, bnd=None):
        u = torch.zeros(self.V, x.shape[1], dtype=torch.float64, device="cuda")
        u[self.inner] = x
        if bnd is not None:
            u[self.outer] = bnd
        return u

    def apply(self, name, bname, u):   # inner rows of an operator with its boundary columns
        return self.mat(name) @ u[self.inner].contiguous() + self.mat(bname) @ u[self.outer].contiguous()

    @staticmethod
    def krylov(A, d, b, rounds=4, eps=1e-14, most=6000):
        """A x = b column by column: Jacobi-preconditioned BiCGStab, restarted from the true residual."""
        x = torch.zeros_like(b)
        bn = b.norm(dim=0).clamp_min(1e-300)
        for _ in range(rounds):
            r = b - A(x)
            if float((r.norm(dim=0) / bn).max()) < eps:
                break
            goal = torch.maximum(1e-9 * r.norm(dim=0), 0.3 * eps * bn)
            dx, rh = torch.zeros_like(b), r.clone()
            rho = alpha = omega = torch.ones_like(bn)
            v = p = torch.zeros_like(b)
            for it in range(most):
                new = (rh * r).sum(0)
                beta = torch.nan_to_num((new / rho) * (alpha / omega), 0.0, 0.0, 0.0)
                rho = new
                p = r + beta * (p - omega * v)
                y = p / d
                v = A(y)
                alpha = torch.nan_to_num(rho / (rh * v).sum(0), 0.0, 0.0, 0.0)
                s = r - alpha * v
                z = s / d
                t = A(z)
                omega = torch.nan_to_num((t * s).sum(0) / (t * t).sum(0), 0.0, 0.0, 0.0)
                more = (r.norm(dim=0) > goal).double()
                dx = dx + more * (alpha * y + omega * z)
                r = torch.where(more > 0, s - omega * t, r)
                if it % 20 == 19 and bool((r.norm(dim=0) <= goal).all()):
                    break
            x = x + dx
        return x

    @staticmethod
    def fixed_point(T, x, most=30):
        """x = T(x) for an affine T: GMRES on the difference of x and T(x), restarted once from the true one."""
        for _ in range(2):
            r = T(x) - x
            base, Q, H = x + r, [r / r.norm()], np.zeros((most + 1, most))
            for k in range(most):
                v = Q[k] - (T(x + r.norm() * Q[k]) - base) / r.norm()
                for _ in range(2):
                    for j, q in enumerate(Q):
                        h = float((q * v).sum())
                        H[j, k] += h
                        v = v - h * q
                H[k + 1, k] = float(v.norm())
                e = np.zeros(k + 2)
                e[0] = float(r.norm())
                y, left = np.linalg.lstsq(H[:k + 2, :k + 1], e, rcond=None)[:2]
                if H[k + 1, k] < 1e-14 or (left.size and math.sqrt(left[0]) < 1e-10 * e[0]):
                    break
                Q.append(v / H[k + 1, k])
            x = x + sum(float(c) * q for c, q in zip(y, Q))
        return x

    def inverse(self, name, b):
        A = self.mat(name)
        return self.krylov(lambda x: A @ x, self.diag(name), b)

    def helmholtz(self, c1, c2, b):   # (c1 M + c2 L) x = b
        M, L = self.mat("idt"), self.mat("lapl")
        return self.krylov(lambda x: c1 * (M @ x) + c2 * (L @ x), c1 * self.diag("idt") + c2 * self.diag("lapl"), b)

    def laplacian(self, u, bnd=None):   # full vector, the boundary value written in
        return self.full(self.inverse("idt", self.apply("lapl", "bnd3", u)), bnd)

    def poisson(self, F, bnd=None):
        b = self.mat("idt") @ F[self.inner].contiguous()
        if bnd is not None:
            b = b + self.mat("bnd2") @ bnd
        return self.full(self.inverse("lapl", b), bnd)

    def jacobian(self, u, v):   # inner points
        k = u.shape[1]
        rhs = [self.apply(n, n + "b", f) for f in (u, v) for n in ("d1", "d2", "d1c", "d2c")]
        x = self.inverse("jidt", torch.cat(rhs, 1))
        a1u, a2u, c1u, c2u, a1v, a2v, c1v, c2v = (x[:, q * k:(q + 1) * k] for q in range(8))
        return 0.25 * ((c2u * a1v - c1u * a2v) + (a2u * c1v - a1u * c2v) + (c2u * a1v - a1u * c2v) + (a2u * c1v - c1u * a2v))

    def norm(self, u):
        return (u * (self.mat("norm") @ u)).sum(0).sqrt()

    def barotropic(self, u):
        tau, sg, mu, th = BV["tau"], BV["sigma"], BV["mu"], BV["theta"]
        M = self.mat("idt")
        w = self.laplacian(u)
        fc = (1 / tau - sg * (1 - th)) * w + mu * (1 - th) * self.laplacian(w)
        un, wn = torch.zeros_like(u), torch.zeros_like(u)
        for _ in range(BV["picard_iters"]):
            J = self.jacobian(th * un + (1 - th) * u,
                              BV["k1"] * (th * wn + (1 - th) * w) + BV["k2"] * self.coriolis)
            wn = self.full(self.helmholtz(1 / tau + sg * th, -th * mu, M @ (fc[self.inner] - J)))
            un = self.poisson(wn)
        return un

    def adjoint(self, v, z):
        tau, sg, mu, th = BV["tau"], BV["sigma"], BV["mu"], BV["theta"]
        lz = self.laplacian(z)
        v = self.poisson(v)
        v = self.full(self.helmholtz(1 / tau + sg * th, -th * mu, self.mat("idt") @ v[self.inner].contiguous()))
        lv = self.laplacian(v)
        jl, jz, jv = (self.full(-self.jacobian(a, b)) for a, b in ((v, self.coriolis), (z, v), (v, lz)))
        h = BV["k1"] * (jv + self.laplacian(jz)) + BV["k2"] * jl
        out = (1 / tau - (1 - th) * sg) * lv + (1 - th) * mu * self.laplacian(lv) - h
        return self.full(out[self.inner])

    def two_layers(self, u1, u2):
        tau, sg, mu, sg1, mu1, al2 = BC["tau"], BC["sigma"], BC["mu"], BC["sigma1"], BC["mu1"], BC["alpha"] ** 2
        th, M, i = 0.5, self.mat("idt"), self.inner
        w1, w2 = self.laplacian(u1), self.laplacian(u2)
        a = 0.5 * (1 - th) * sg
        f = -a * w1 + a * w2 + mu * (1 - th) * self.laplacian(w1) + w1 / tau
        g = -a * w1 - a * w2 + mu * (1 - th) * self.laplacian(w2) + w2 / tau \
            - al2 / tau * u2 - al2 * mu1 * (1 - th) * w2 + al2 * sg1 * (1 - th) * u2
        un1, un2, wn1, wn2 = u1, u2, w1, w2
        for _ in range(BC["picard_iters"]):
            U1, U2 = (1 - th) * u1 + th * un1, (1 - th) * u2 + th * un2
            W1, W2 = (1 - th) * w1 + th * wn1 + self.coriolis, (1 - th) * w2 + th * wn2
            J = [self.jacobian(p, q) for p, q in ((U1, W1), (U2, W2), (U1, W2), (U2, W1), (U1, U2))]
            r1 = M @ (f[i] - J[0] - J[1])
            r2 = M @ (g[i] - J[2] - J[3] + al2 * J[4])
            # the block system, reduced to w2: given w2, u2 = L^-1 M w2, then w1 and w2 by their mass-like blocks

            def upper(x2):
                return self.helmholtz(1 / tau + 0.5 * th * sg, -th * mu, r1 + 0.5 * sg * th * (M @ x2))

            def sweep(x2):
                return self.helmholtz(1 / tau + 0.5 * th * sg + al2 * th * mu1, -th * mu,
                                      r2 - 0.5 * sg * th * (M @ upper(x2))
                                      + (al2 / tau + al2 * th * sg1) * (M @ self.inverse("lapl", M @ x2)))

            x2 = self.fixed_point(sweep, wn2[i])
            x1, s2 = upper(x2), self.inverse("lapl", M @ x2)
            wn1, wn2 = self.full(x1), self.full(x2)
            b1, b2 = self.full(self.inverse("lapl", M @ x1)), self.full(s2)
            far = max(float(self.norm(b1 - un1)), float(self.norm(b2 - un2)))
            un1, un2 = b1, b2
            if far < BC["picard_tol"]:
                break
        return un1, un2


@functools.lru_cache(maxsize=None)
def _discrete(level):
    return _Discrete(level)


def exact(case, seed):
    kind, level, members = case["kind"], case["level"], case["members"]
    if kind in ("step", "run") and members * case["steps"] * 4 ** level > 64 * 4 ** 6:
        return None   # over 20 seconds
    D, x = _discrete(level), _inputs(case, seed)
    if kind == "mult32":
        return D.mat("lapl") @ x["x"].double()
    if kind == "solve":
        return D.poisson(x["F"].T.contiguous(), x["bnd"].T.contiguous()).T
    if kind == "laplacian":
        return D.laplacian(x["u"][:, None])[:, 0]
    if kind == "jacobian":
        return D.full(D.jacobian(x["u"][:, None], x["v"][:, None]))[:, 0]
    if kind == "adjoint":
        return D.adjoint(x["u"][:, None], x["z"][:, None])[:, 0]
    if kind == "baroclin":
        return torch.cat(D.two_layers(x["u1"][:, None], x["u2"][:, None]), 1).T
    u = x["u"].T.contiguous()
    for _ in range(case["steps"]):
        u = D.barotropic(u)
    return u.T
