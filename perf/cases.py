"""The work that programs built on this framework have it do, as cases to be measured.

A case is a dict of plain values.  `kind` names the public entry point that one pass goes through:

* `matvec`   VoxelOperator.matvec: y = K(E) u, with or without the Dirichlet mask; float64, float32
             or bfloat16 storage.
* `sweep`    VoxelOperator.jacobi: one damped-Jacobi smoothing step.
* `vcycle`   MGHierarchy.emit: one V(2,2) cycle applied to a residual.
* `solve`    ElasticitySolver.solve: a whole solve on the device (Jacobi-PCG or GMG-PCG to 1e-8).
* `host`     voxel_b200.solve: host arrays in and out, set-up refreshed from the new moduli.
* `simp`     one topology-optimisation step: compliance and its gradient through autograd, the
             sensitivity filter, the optimality-criteria update and the density filter.

Shapes are voxel grids (elements in x, y, z); `exact` restates every entry point in plain FP64 torch.
"""
import math

import numpy as np
import torch

import voxel_b200 as vx
from voxel_b200.problems import cantilever_equal_split

DTYPES = {"f64": torch.float64, "f32": torch.float32, "bf16": torch.bfloat16}
EMIN, PENAL, OMEGA, CHECK_EVERY = 1e-9, 3.0, 0.6, 5
VOLFRAC, RMIN, MOVE, OC_TOL = 0.3, 1.5, 0.2, 1e-6


def listed():
    return [
        # the smallest operator call (28,611 DOF, the Jacobi-PCG benchmark's grid): launch latency
        dict(name="matvec_f64_32x16x16", kind="matvec", nx=32, ny=16, nz=16, dtype="f64", masked=True),
        # the FP64 operator of a mid-size grid (12.8M DOF), as an outside Krylov loop calls it
        dict(name="matvec_f64_256x128x128", kind="matvec", nx=256, ny=128, nz=128, dtype="f64", masked=True),
        # an odd grid in FP32 without constraints: ragged tiles in every direction
        dict(name="matvec_f32_203x97x131", kind="matvec", nx=203, ny=97, nz=131, dtype="f32", masked=False),
        # the largest grid with bf16 storage
        dict(name="matvec_bf16_576x288x288", kind="matvec", nx=576, ny=288, nz=288, dtype="bf16", masked=True),
        # one preconditioner application on the small benchmark grid, FP32
        dict(name="vcycle_f32_128x64x64", kind="vcycle", nx=128, ny=64, nz=64, dtype="f32"),
        # one on the mid-size serving grid, FP64
        dict(name="vcycle_f64_160x80x80", kind="vcycle", nx=160, ny=80, nz=80, dtype="f64"),
        # the smallest whole solve: FP64 Jacobi-PCG, hundreds of short iterations
        dict(name="solve_jacobi_32x16x16", kind="solve", nx=32, ny=16, nz=16, precision="jacobi"),
        # the small GMG benchmark in plain FP64
        dict(name="solve_fp64_128x64x64", kind="solve", nx=128, ny=64, nz=64, precision="fp64"),
        # a bf16-storage preconditioner on the largest serving grid
        dict(name="solve_bf16_256x128x128", kind="solve", nx=256, ny=128, nz=128, precision="bf16"),
        # the headline: 144.6M DOF, mixed precision
        dict(name="solve_mixed_576x288x288", kind="solve", nx=576, ny=288, nz=288, precision="mixed"),
        # a request with host buffers on the small GMG grid: copies, refresh, coarse factor, solve
        dict(name="host_mixed_128x64x64", kind="host", nx=128, ny=64, nz=64, precision="mixed"),
        # one step of the topology-optimisation benchmark
        dict(name="simp_step_192x96x96", kind="simp", nx=192, ny=96, nz=96, precision="mixed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mg_shape(rng, most):
    """A grid that coarsens to at most 16 elements in x: coarsest extents times a power of two."""
    while True:
        c = (rng.randint(9, 16), rng.randint(3, 9), rng.randint(3, 9))
        f = 2 ** rng.randint(1, 5)
        nx, ny, nz = (v * f for v in c)
        if 2000 <= nx * ny * nz <= most:
            return nx, ny, nz


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "sweep", "vcycle", "vcycle", "solve", "solve", "host", "simp"])
    if kind in ("matvec", "sweep"):
        while True:
            nx, ny, nz = (_log_int(rng, lo, hi) for lo, hi in ((16, 600), (8, 300), (8, 300)))
            if nx * ny * nz <= 576 * 288 * 288:
                break
        dtype = rng.choice(["f64", "f32", "bf16"] if kind == "matvec" else ["f64", "f32"])
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=dtype, masked=kind == "sweep" or rng.random() < 0.7)
    if kind == "vcycle":
        nx, ny, nz = _mg_shape(rng, 30_000_000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=rng.choice(["f32", "f32", "f64"]))
    if kind == "solve":
        if rng.random() < 0.2:
            return dict(kind=kind, nx=_log_int(rng, 16, 48), ny=_log_int(rng, 8, 24), nz=_log_int(rng, 8, 24),
                        precision="jacobi")
        nx, ny, nz = _mg_shape(rng, 12_000_000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=rng.choice(["mixed", "mixed", "bf16", "fp64"]))
    if kind == "host":
        nx, ny, nz = _mg_shape(rng, 4_000_000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=rng.choice(["mixed", "mixed", "fp64"]))
    nx, ny, nz = _mg_shape(rng, 3_000_000)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision="mixed")


def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _ke():
    return vx.quadrature([1.0, 1.0, 1.0], 0.3)


def _density(shape, seed, ell=8.0):
    """A correlated density field in [1e-3, 1]: white noise smoothed over `ell` voxels, mapped through a
    logistic (the benchmark workloads' field)."""
    w = torch.randn(shape, dtype=torch.float64, device="cuda", generator=_gen(seed))
    k = [torch.fft.fftfreq(n, dtype=torch.float64, device="cuda") ** 2 for n in shape]
    w = torch.fft.fftn(w)
    for ax, k2 in enumerate(k):
        w *= torch.exp(-2 * math.pi ** 2 * ell ** 2 * k2).reshape([-1 if a == ax else 1 for a in range(3)])
    g = torch.fft.ifftn(w).real
    g = (g - g.mean()) / g.std(correction=0)
    return (1e-3 + (1 - 1e-3) / (1 + torch.exp(-g))).reshape(-1).contiguous()


def _modulus(shape, seed):
    """The moduli of the benchmark workloads' density fields: uniform on the smallest grids, else correlated."""
    if shape[0] * shape[1] * shape[2] < 20000:
        rho = 0.01 + 0.99 * torch.rand(int(np.prod(shape)), dtype=torch.float64, device="cuda", generator=_gen(seed))
    else:
        rho = _density(shape, seed)
    return EMIN + (1.0 - EMIN) * rho ** PENAL


def _vector(shape, seed):
    return torch.randn(3 * vx.n_nodes(shape), dtype=torch.float64, device="cuda", generator=_gen(seed + 7919))


def _design(shape, seed):
    """A design part of the way through an optimisation: void, solid and grey regions of mean VOLFRAC."""
    rho = _density(shape, seed, 6.0)
    x = torch.clamp(0.5 + 1.5 * (rho - rho.mean()), 0.05, 1.0)
    return torch.clamp(x * (VOLFRAC / x.mean()), 0.01, 1.0)


def prepare(case, seed):
    shape, kind = _shape(case), case["kind"]
    if kind in ("matvec", "sweep"):
        dt = DTYPES[case["dtype"]]
        op = vx.VoxelOperator(shape, _ke(), dt)
        s = dict(op=op, E=_modulus(shape, seed).to(dt), u=_vector(shape, seed).to(dt), mask=None)
        if case["masked"]:
            s["mask"] = vx.node_mask_from_dofs(cantilever_equal_split(shape)[0])
        if kind == "sweep":
            s["r"] = _vector(shape, seed + 1).to(dt)
            s["invd"] = op.diagonal(s["E"], s["mask"], inverse=True)
        s["out"] = torch.empty(op.ndof, dtype=torch.float32 if dt == torch.bfloat16 else dt, device="cuda")
        return s
    mask, force = cantilever_equal_split(shape)
    if kind == "vcycle":
        M = vx.MGHierarchy(shape, _ke(), _modulus(shape, seed), vx.node_mask_from_dofs(mask), DTYPES[case["dtype"]],
                           2, 2, OMEGA)
        return dict(M=M, r=_vector(shape, seed) * mask)
    if kind == "solve":
        s = vx.ElasticitySolver(shape, _modulus(shape, seed), mask, precision=case["precision"], tol=1e-8,
                                maxiter=5000 if case["precision"] == "jacobi" else 200, omega=OMEGA,
                                check_every=50 if case["precision"] == "jacobi" else CHECK_EVERY)
        return dict(solver=s, f=force)
    if kind == "host":
        pin = lambda t: t.cpu().pin_memory()
        return dict(shape=shape, E=pin(_modulus(shape, seed)), f=pin(force), mask=pin(mask), precision=case["precision"],
                    out=torch.empty(force.numel(), dtype=torch.float64).pin_memory())
    x = _design(shape, seed)
    filt = vx.ConeFilter(*shape, RMIN)
    rho = filt.forward(x)
    solver = vx.ElasticitySolver(shape, vx.simp_modulus(rho, EMIN, 1.0, PENAL), mask, precision=case["precision"],
                                 omega="spectral", tol=1e-6, maxiter=500, check_every=CHECK_EVERY)
    # the displacement that a loop carries over from its previous design
    before = filt.forward(torch.clamp(x + 0.02 * (torch.rand(x.shape, dtype=x.dtype, device="cuda",
                                                             generator=_gen(seed + 1)) - 0.5), 0.0, 1.0))
    solver.update_modulus(vx.simp_modulus(before, EMIN, 1.0, PENAL))
    u0 = solver.solve(force).x.clone()
    return dict(x=x, rho=rho, filt=filt, oc=vx.OCUpdater(filt), u0=u0, state=vx.simp.SimpState(solver, force, EMIN, 1.0, PENAL),
                dv=filt.transpose(torch.ones_like(x)))


def run(s):
    if "op" in s:
        if "r" in s:
            return s["op"].jacobi(s["u"], s["r"], s["invd"], s["E"], s["mask"], OMEGA, out=s["out"])
        return s["op"].matvec(s["u"], s["E"], s["mask"], out=s["out"])
    if "M" in s:
        return s["M"].emit(s["r"])
    if "solver" in s:
        res = s["solver"].solve(s["f"])
        return dict(x=res.x, iterations=res.iterations, converged=res.converged)
    if "out" in s:
        u, info = vx.solve(s["shape"], s["E"], s["f"], s["mask"], precision=s["precision"], check_every=CHECK_EVERY,
                           omega=OMEGA, out=s["out"])
        return dict(x=u, iterations=info["iterations"], compliance=np.float64(info["compliance"]))
    st = s["state"]
    st.u = s["u0"]
    rho = s["rho"].clone().requires_grad_(True)
    c = vx.compliance(rho, st)
    c.backward()
    x_new = s["oc"](s["x"], s["filt"].transpose(rho.grad), s["dv"], VOLFRAC, MOVE, tol=OC_TOL)
    return dict(c=c.detach(), u=st.u, grad=rho.grad, x=x_new, rho=s["filt"].forward(x_new))


def work(case):
    """One read of every input and one write of every output; a solve reads its vectors once an iteration
    (about 20 with multigrid, 500 with Jacobi).  150 operations an element and operator application."""
    nx, ny, nz = _shape(case)
    n, ne = (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz
    kind = case["kind"]
    if kind in ("matvec", "sweep"):
        w = {"f64": 8, "f32": 4, "bf16": 2}[case["dtype"]]
        out = max(w, 4)
        b = (3 * w + 3 * out + case["masked"]) * n + w * ne + (6 * w * n if kind == "sweep" else 0)
        return {"bytes": b, "flops": 150 * ne}
    if kind == "vcycle":
        w = 8 if case["dtype"] == "f64" else 4
        return {"bytes": (24 + 3 * w + 1) * n + w * ne, "flops": 8 / 7 * 5 * 150 * ne}
    its, apps = (500, 1) if case.get("precision") == "jacobi" else (20, 7)
    b = (48 + 1) * n + 8 * ne
    return {"bytes": its * b, "flops": its * apps * 150 * ne}


# ----------------------------------------------------------------------------- plain FP64 restatement
_CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


class _Op:
    """K(E), its Dirichlet form and its diagonal by gathering each element's 24 values."""

    def __init__(self, shape, ke, E, mask):
        self.s, self.E, self.m = shape, E.reshape(shape), mask
        self.k = torch.as_tensor(ke, dtype=torch.float64, device="cuda")
        self.nodes = tuple(v + 1 for v in shape) + (3,)

    def raw(self, u):
        nx, ny, nz = self.s
        u, y = u.reshape(self.nodes), torch.zeros(self.nodes, dtype=torch.float64, device="cuda")
        step = max(1, 4_000_000 // (ny * nz))
        for a in range(0, nx, step):
            b = min(nx, a + step)
            at = [(slice(a + i, b + i), slice(j, j + ny), slice(k, k + nz)) for i, j, k in _CORNERS]
            ue = torch.cat([u[c] for c in at], dim=3) * self.E[a:b, :, :, None]
            f = ue @ self.k.T
            for i, c in enumerate(at):
                y[c] += f[..., 3 * i:3 * i + 3]
        return y.reshape(-1)

    def __call__(self, u):
        return self.raw(u) if self.m is None else self.m * self.raw(self.m * u) + (1 - self.m) * u

    def energy(self, u):
        nx, ny, nz = self.s
        u, e = u.reshape(self.nodes), torch.empty(self.s, dtype=torch.float64, device="cuda")
        for a in range(nx):
            ue = torch.cat([u[a + i, j:j + ny, k:k + nz] for i, j, k in _CORNERS], dim=2)
            e[a] = ((ue @ self.k.T) * ue).sum(2)
        return e.reshape(-1)

    def inverse_diagonal(self):
        nx, ny, nz = self.s
        d = torch.zeros(self.nodes, dtype=torch.float64, device="cuda")
        kd = self.k.diagonal()
        for n, (i, j, k) in enumerate(_CORNERS):
            d[i:i + nx, j:j + ny, k:k + nz] += self.E[..., None] * kd[3 * n:3 * n + 3]
        d = d.reshape(-1)
        return 1 / d if self.m is None else 1 / torch.where(self.m > 0, d, torch.ones_like(d))

    def dense(self):
        nx, ny, nz = self.s
        n = self.nodes[0] * self.nodes[1] * self.nodes[2]
        node = torch.arange(n, device="cuda").reshape(self.nodes[:3])
        conn = torch.stack([node[i:i + nx, j:j + ny, k:k + nz].reshape(-1) for i, j, k in _CORNERS], dim=1)
        dof = (3 * conn[:, :, None] + torch.arange(3, device="cuda")).reshape(-1, 24)
        A = torch.zeros(3 * n, 3 * n, dtype=torch.float64, device="cuda")
        A.index_put_((dof[:, :, None].expand(-1, 24, 24), dof[:, None, :].expand(-1, 24, 24)),
                     self.E.reshape(-1, 1, 1) * self.k, accumulate=True)
        A = self.m[:, None] * A * self.m
        A.diagonal().add_(1 - self.m)
        return A


def _restrict(r, fine):
    v = r.reshape(tuple(s + 1 for s in fine) + (3,))
    for ax in range(3):
        n = fine[ax] // 2
        c = v.index_select(ax, 2 * torch.arange(n + 1, device="cuda"))
        o = 0.5 * v.index_select(ax, 2 * torch.arange(n, device="cuda") + 1)
        c.narrow(ax, 0, n).add_(o)
        c.narrow(ax, 1, n).add_(o)
        v = c
    return v.reshape(-1)


def _prolong(e, fine):
    v = e.reshape(tuple(s // 2 + 1 for s in fine) + (3,))
    for ax in range(3):
        n = v.shape[ax] - 1
        mid = 0.5 * (v.narrow(ax, 0, n) + v.narrow(ax, 1, n))
        both = torch.stack([v.narrow(ax, 0, n), mid], dim=ax + 1)
        shape = list(v.shape)
        shape[ax] = 2 * n
        v = torch.cat([both.reshape(shape), v.narrow(ax, n, 1)], dim=ax)
    return v.reshape(-1)


class _Cycle:
    def __init__(self, shape, ke, E, mask):
        self.ops, self.invd, self.shapes = [], [], vx.hierarchy_shapes(shape, 16)
        for i, s in enumerate(self.shapes):
            if i:
                nx, ny, nz = s
                E = E.reshape(nx, 2, ny, 2, nz, 2).mean(dim=(1, 3, 5)).reshape(-1)
                p = tuple(v + 1 for v in self.shapes[i - 1]) + (3,)
                mask = mask.reshape(p)[::2, ::2, ::2].reshape(-1)
            self.ops.append(_Op(s, ke * 2 ** i, E, mask))
            self.invd.append(self.ops[-1].inverse_diagonal())
        self.L = torch.linalg.cholesky(self.ops[-1].dense())

    def __call__(self, r, i=0):
        A, d = self.ops[i], self.invd[i]
        if i == len(self.ops) - 1:
            return torch.cholesky_solve((A.m * r)[:, None], self.L)[:, 0] * A.m
        x = OMEGA * d * r
        x = x + OMEGA * d * (r - A(x))
        rc = _restrict((r - A(x)) * A.m, self.shapes[i]) * self.ops[i + 1].m
        x = x + _prolong(self(rc, i + 1), self.shapes[i]) * A.m
        for _ in range(2):
            x = x + OMEGA * d * (r - A(x))
        return x


def _solution(shape, E, mask, f, jacobi=False):
    """A x = f to near rounding by preconditioned CG in FP64."""
    A = _Op(shape, _ke(), E, mask)
    if jacobi:
        d = A.inverse_diagonal()
        M = lambda r: d * r
    else:
        M = _Cycle(shape, _ke(), E, mask)
    x, r, nb, p, rz, z_old = torch.zeros_like(f), f.clone(), float(f.norm()), None, None, None
    for k in range(6000 if jacobi else 120):
        z = M(r)
        rzn = torch.dot(r, z)
        p = z if p is None else z + (torch.dot(r, z - z_old) / rz) * p
        rz, z_old = rzn, z
        q = A(p)
        a = rz / torch.dot(p, q)
        x = x + a * p
        r = r - a * q
        if k % (100 if jacobi else 5) == 0:
            r = f - A(x)
            if float(r.norm()) <= 1e-13 * nb:
                break
    return x


def _filter(shape, v, transpose):
    def H(a):
        a, y = a.reshape(shape), torch.zeros(shape, dtype=torch.float64, device="cuda")
        R = int(math.ceil(RMIN)) - 1
        for o in np.ndindex(2 * R + 1, 2 * R + 1, 2 * R + 1):
            o = [i - R for i in o]
            w = RMIN - math.sqrt(sum(i * i for i in o))
            if w > 0:
                dst = tuple(slice(max(0, -i), n - max(0, i)) for i, n in zip(o, shape))
                src = tuple(slice(max(0, i), n - max(0, -i)) for i, n in zip(o, shape))
                y[dst] += w * a[src]
        return y.reshape(-1)
    s = H(torch.ones_like(v))
    return H(v / s) if transpose else H(v) / s


def exact(case, seed):
    shape, kind = _shape(case), case["kind"]
    if kind in ("matvec", "sweep"):
        s = prepare(case, seed)
        m = cantilever_equal_split(shape)[0] if case["masked"] else None
        E, u = s["E"].double(), s["u"].double()
        y = _Op(shape, _ke(), E, m)(u)
        return y if kind == "matvec" else u + OMEGA * s["invd"].double() * (s["r"].double() - y)
    mask, force = cantilever_equal_split(shape)
    if kind == "simp":
        x = _design(shape, seed)
        rho = _filter(shape, x, False)
        E = EMIN + (1 - EMIN) * rho ** PENAL
        u = _solution(shape, E, mask, force)
        grad = -PENAL * rho ** (PENAL - 1) * (1 - EMIN) * _Op(shape, _ke(), E, mask).energy(u)
        dc, dv = _filter(shape, grad, True), _filter(shape, torch.ones_like(x), True)
        l1, l2 = 0.0, 1e9
        while (l2 - l1) / (l1 + l2) > OC_TOL:
            mid = 0.5 * (l1 + l2)
            xn = x * torch.sqrt(torch.clamp(-dc / dv / mid, min=0))
            xn = torch.minimum(torch.maximum(xn, torch.clamp(x - MOVE, min=0)), torch.clamp(x + MOVE, max=1))
            if float(_filter(shape, xn, False).mean()) > VOLFRAC:
                l1 = mid
            else:
                l2 = mid
        return dict(c=torch.dot(force, u), u=u, grad=grad, x=xn, rho=_filter(shape, xn, False))
    E = _modulus(shape, seed)
    if kind == "vcycle":
        return _Cycle(shape, _ke(), E, mask)(_vector(shape, seed) * mask)
    x = _solution(shape, E, mask, force, case["precision"] == "jacobi")
    if kind == "host":
        return dict(x=x, iterations=None, compliance=np.float64(float(torch.dot(force, x))))
    return dict(x=x, iterations=None, converged=None)
