"""The calls whose speed is measured, over the range that users of the library run.

A case is one call through the public entry points (`Context`, `autograd`, `batch`) on a grid of
n^3 voxels:

  apply_d    D u = div(k grad u)
  diffusion  one Crank-Nicolson step (PCG with the spectral preconditioner)
  smooth     the Weierstrass smoother
  forward    c(0) -> c(1)
  adjoint    forward, then the discrete adjoint of a given cotangent (torch autograd)
  gradient   objective and gradient over (p, kappa, rho) (torch autograd)
  hessian    Gauss-Newton matvec over p
  batch      the gradients of several uneven problems as one CUDA graph

Grids: 16^3 to 256^3. 64^3, 128^3 and 256^3 are the sizes of the workloads in bench.py and the
tests, 32^3 and 16^3 those of quick studies; images resampled at another voxel size give any other
multiple of 8 (what the library takes) in between. "fp64" is a context with all fields in double,
"mixed" one with float fields; a mixed context is fed float32 tensors, as the torch programs
around it hold them, and its results are float32.
"""
import math

import numpy as np
import torch

from glia_gb300 import _abi, native, synthetic
from glia_gb300.autograd import rd_objective, solve_state
from glia_gb300.batch import Batch, GraphBatch, Problem
from glia_gb300.context import Context

DT = 0.01
SIGMA = 2 * math.pi / 64   # width of the Gaussian basis functions on grids that resolve it
GM = 0.2                   # grey-matter diffusivity relative to white matter
EVERY = 10                 # steps between checkpoints

# Work of one pass relative to a mixed PCG solve on one voxel, for keeping draws affordable.
SOLVES = {"apply_d": lambda nt: 0.3, "smooth": lambda nt: 0.3, "diffusion": lambda nt: 1,
          "forward": lambda nt: 2 * nt, "adjoint": lambda nt: 4 * nt,
          "gradient": lambda nt: 6 * nt, "hessian": lambda nt: 4 * nt}


def listed():
    def case(name, op, n, precision, nt=1, gaussians=0, kappa=0.02, rho=8.0, small=0):
        return {"name": name, "op": op, "n": n, "precision": precision, "nt": nt,
                "gaussians": gaussians, "kappa": kappa, "rho": rho, "small": small}

    return [
        # one operator apply on the smallest usual grid: launches and latency
        case("apply_d_fp64_32", "apply_d", 32, "fp64"),
        # the plain forward simulation: one tumour, 100 steps, double precision (the default)
        case("forward_fp64_64", "forward", 64, "fp64", nt=100, kappa=0.05, rho=10.0),
        # an image resampled to a size that is no power of two, both precisions
        case("forward_mixed_96", "forward", 96, "mixed", nt=20),
        case("adjoint_fp64_120", "adjoint", 120, "fp64", nt=2),
        # a diffusion step at full resolution in double precision
        case("diffusion_fp64_256", "diffusion", 256, "fp64"),
        # the evaluation an inversion repeats, from a quick study to full resolution
        case("gradient_mixed_32", "gradient", 32, "mixed", nt=16, gaussians=8),
        case("gradient_mixed_64", "gradient", 64, "mixed", nt=40, gaussians=64),
        case("gradient_mixed_128", "gradient", 128, "mixed", nt=40, gaussians=216, kappa=0.03,
             rho=12.0),
        case("gradient_mixed_256", "gradient", 256, "mixed", nt=20, gaussians=512),
        # the same in double precision
        case("gradient_fp64_128", "gradient", 128, "fp64", nt=6, gaussians=216, kappa=0.03,
             rho=12.0),
        # a Newton-Krylov inversion's matvec
        case("hessian_fp64_64", "hessian", 64, "fp64", nt=10, gaussians=64),
        # several patients at once: 2 problems on n^3, 6 on small^3
        case("batch_mixed", "batch", 128, "mixed", nt=10, gaussians=216, small=64),
    ]


def draw(rng):
    largest = 1.01 * 256 ** 3 * SOLVES["gradient"](20)
    while True:
        op = rng.choice(["apply_d", "diffusion", "smooth", "forward", "forward", "adjoint",
                         "gradient", "gradient", "gradient", "hessian", "batch"])
        precision = ("fp64" if op == "hessian" else "mixed" if op == "batch"
                     else rng.choice(["fp64", "mixed", "mixed"]))
        usual = rng.random() < 0.6
        n = rng.choice([32, 64, 128, 256]) if usual else 8 * round(2 * 16 ** rng.random())
        nt = 1 if op in ("apply_d", "diffusion", "smooth") else round(2 * 50 ** rng.random())
        small = 0
        if op == "batch":
            n, small, nt = rng.choice([(128, 64), (96, 48), (64, 32), (128, 32)]) + (
                rng.randint(4, 12),)
        gaussians = 0
        if op in ("gradient", "hessian", "batch"):
            gaussians = {32: 8, 64: 64, 128: 216, 256: 512}.get(n, max(4, n * n // 80))
        cost = n ** 3 * SOLVES["gradient" if op == "batch" else op](nt)
        cost *= 25 if precision == "fp64" else 2.5 if op == "batch" else 1
        if cost <= largest:
            return {"op": op, "n": n, "precision": precision, "nt": nt, "gaussians": gaussians,
                    "kappa": round(0.01 * 6 ** rng.random(), 4),
                    "rho": round(4 + 10 * rng.random(), 3), "small": small}


# ---- inputs ---------------------------------------------------------------------------------

def axis(n):
    return torch.arange(n, device="cuda", dtype=torch.float64) * (2 * math.pi / n)


def weierstrass(n, sigma):
    """The smoother along one axis: the circulant matrix of the periodised Gaussian."""
    d = axis(n)
    w = torch.exp(-(d / sigma) ** 2 / 2) + torch.exp(-((d - 2 * math.pi) / sigma) ** 2 / 2)
    i = torch.arange(n, device="cuda")
    return (w / w.sum())[(i[:, None] - i[None, :]) % n]


def along_axes(f, mx, my, mz):
    f = torch.einsum("xyz,cz->xyc", f, mz)
    f = torch.einsum("xyc,by->xbc", f, my)
    return torch.einsum("xbc,ax->abc", f, mx)


def smoothed(f, sigma):
    w = weierstrass(f.shape[0], sigma)
    return along_axes(f, w, w, w)


def tissue(n, gen):
    """(wm, gm, csf) in an ellipsoidal brain, made as synthetic.make_tissue makes them."""
    h = 2 * math.pi / n
    x = axis(n) - math.pi
    r = ((x / (0.8 * math.pi))[:, None, None] ** 2 + (x / (0.7 * math.pi))[None, :, None] ** 2
         + (x / (0.6 * math.pi))[None, None, :] ** 2)
    mask = r <= 1
    xi = smoothed(torch.randn((n, n, n), generator=gen, device="cuda", dtype=torch.float64),
                  2 * h)
    lo, hi = xi[mask].min(), xi[mask].max()
    xi = (xi - lo) / (hi - lo)
    classes = (mask & (xi > 0.75), mask & (xi > 0.45) & (xi <= 0.75), mask & (xi <= 0.45))
    return [smoothed(m.double(), h) for m in classes]


def bumps(n, at, width):
    """Sum of Gaussians of the given width (in radians) around the points `at`."""
    x, out = axis(n), torch.zeros((n, n, n), device="cuda", dtype=torch.float64)
    for c in at:
        g = [torch.exp(-((x - float(v)) / width) ** 2 / 2) for v in c]
        out += g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :]
    return out


def inputs(case, seed, n):
    """Everything one problem is made of, as float64 tensors on the GPU and numpy vectors."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    real = torch.float64 if case["precision"] == "fp64" else torch.float32
    wm, gm, csf = tissue(n, gen)
    h = 2 * math.pi / n
    p = {"n": n, "wm": wm, "gm": gm, "csf": csf, "sigma": max(SIGMA, h), "real": real}
    inside = np.array([math.pi] * 3) + rng.uniform(-0.3, 0.3, (3, 3)) * math.pi
    # a tumour at t = 0, a cotangent at t = 1 and a segmented image of a later tumour
    p["c0"] = bumps(n, inside[:1], max(SIGMA, 1.5 * h)).to(real)
    p["g"] = (bumps(n, inside, 0.5) * torch.randn((n, n, n), generator=gen, device="cuda",
                                                  dtype=torch.float64)).to(real)
    p["d1"] = (bumps(n, inside, 0.4) > 0.5).to(real)
    if case["gaussians"]:
        region = (wm + gm > 0.5).cpu().numpy()
        # centres off the voxels, so that no voxel sits on the basis functions' cut at 5 sigma
        p["centers"] = synthetic.lattice_centers_in_mask(
            region, min(case["gaussians"], int(region.sum()))) + 0.013 * h
        count = len(p["centers"])
        active = rng.choice(count, max(1, round(0.05 * count)), replace=False)
        coef = np.zeros(count)
        coef[active] = rng.uniform(0.2, 1.0, active.size)
        p["x"] = np.concatenate([coef, [case["kappa"], case["rho"]]]).astype(
            np.float64 if real == torch.float64 else np.float32)
        p["direction"] = np.concatenate([rng.standard_normal(count), [0.0, 0.0]])
    return p


def context(case, p, every=0):
    ctx = Context(native.load(), p["n"], _abi.GLIA_FP64 if p["real"] == torch.float64
                  else _abi.GLIA_MIXED)
    ctx.set_pointer_mode(_abi.GLIA_PTR_DEVICE_F64)
    torch.cuda.synchronize()
    ctx.set_time(DT, case["nt"])
    # the preconditioner of the Strang half step, which every solve after the first runs with
    ctx.set_pcg(pc_dt_mode=_abi.GLIA_PC_DT_FIXED, pc_dt=DT / 2)
    ctx.set_tissue(*(t.reshape(-1) for t in (p["wm"], p["gm"], p["csf"])))
    ctx.set_coefficients(k=case["kappa"], rho=case["rho"], k_gm_wm=GM)
    if case["op"] in ("gradient", "hessian"):
        ctx.set_phi(p["centers"], p["sigma"])
        ctx.set_opt(np=len(p["centers"]), nk=1, nr=1, diffusivity_inversion=0, beta=0.0,
                    all_gradients=1)
    if every:
        ctx.set_history(_abi.GLIA_HISTORY_CHECKPOINT, every)
    elif case["op"] == "forward":
        ctx.set_history(_abi.GLIA_HISTORY_OFF)
    ctx.set_pointer_mode(_abi.GLIA_PTR_DEVICE_F64 if p["real"] == torch.float64
                         else _abi.GLIA_PTR_DEVICE_F32)
    return ctx


def prepare(case, seed):
    if case["op"] == "batch":
        return prepare_batch(case, seed)
    p = inputs(case, seed, case["n"])
    ctx = context(case, p, EVERY if case["op"] == "gradient" else 0)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    s = {"op": case["op"], "ctx": ctx, "stream": stream, "c0": p["c0"], "g": p["g"]}
    if case["op"] == "gradient":
        s["x"] = torch.from_numpy(p["x"]).requires_grad_()
        s["d1"] = p["d1"].reshape(-1)
    elif case["op"] == "hessian":
        s["direction"] = p["direction"]
        ctx.eval_objective_and_gradient(p["x"], p["d1"].reshape(-1))
    elif case["op"] in ("apply_d", "smooth"):
        s["out"] = torch.empty_like(p["c0"].reshape(-1))
    torch.cuda.synchronize()
    return s


def batch_problems(case, seed):
    out = []
    for b, n in enumerate([case["n"]] * 2 + [case["small"]] * 6):
        gaussians = case["gaussians"] if n == case["n"] else {32: 8, 64: 64}.get(n, 28)
        kappa, rho = case["kappa"] * (1 + 0.05 * b), case["rho"] * (1 - 0.03 * b)
        out.append(({**case, "gaussians": gaussians, "kappa": kappa, "rho": rho}, n,
                    1000 * seed + b))
    return out


class OwnedGraph(GraphBatch):
    """A captured batch that goes with its contexts when it is dropped."""

    def __del__(self):
        self.close()
        self.batch.close()


def prepare_batch(case, seed):
    problems, data = [], []
    for sub, n, sub_seed in batch_problems(case, seed):
        p = inputs(sub, sub_seed, n)
        wl = synthetic.GradientWorkload(n=n, nt=sub["nt"], dt=DT, n_gauss=len(p["centers"]),
                                        rho=sub["rho"], kappa=sub["kappa"], k_gm_wm=GM,
                                        sigma=p["sigma"])
        maps = [t.cpu().numpy() for t in (p["wm"], p["gm"], p["csf"])]
        ti = synthetic.Tissue(*maps, vt=np.zeros_like(maps[0]), mask=maps[0] > 0)
        problems.append(Problem(n, sub["nt"], wl, ti, p["centers"], p["x"].astype(np.float64),
                                sub_seed))
        data.append(p["d1"].cpu().numpy().astype(np.float64).reshape(-1))
    batch = Batch(problems, every=EVERY)
    batch.data = data
    for ctx, pr in zip(batch.ctxs, problems):
        ctx.set_pcg(pc_dt_mode=_abi.GLIA_PC_DT_FIXED, pc_dt=DT / 2)
        ctx.set_launch_geometry(*((2, 1) if pr.n <= 64 else (8, 4)))
    return {"op": "batch", "graph": OwnedGraph(batch)}


# ---- one pass -------------------------------------------------------------------------------

def run(state):
    op = state["op"]
    if op == "batch":
        graph = state["graph"]
        graph.capture()  # every step of the inversions has new parameters, and its own capture
        return [(J, torch.from_numpy(dJ).float()) for J, dJ in graph.evaluate()[1]]
    ctx = state["ctx"]
    if op == "hessian":
        return ctx.hessian_matvec(state["direction"])
    with torch.cuda.stream(state["stream"]):
        if op == "apply_d":
            return ctx.apply_d(state["c0"].reshape(-1), state["out"])
        if op == "smooth":
            return ctx.smooth(state["g"].reshape(-1), 2 * 2 * math.pi / ctx.n, state["out"])
        if op == "diffusion":
            c = state["c0"].reshape(-1).clone()
            ctx.diffusion_solve(c, DT / 2)
            return c
        if op == "forward":
            return solve_state(state["c0"], ctx)
        if op == "adjoint":
            c0 = state["c0"].detach().requires_grad_()
            c1 = solve_state(c0, ctx)
            return c1.detach(), torch.autograd.grad(c1, c0, state["g"])[0]
        J = rd_objective(state["x"], ctx, state["d1"])
        return J.detach(), torch.autograd.grad(J, state["x"])[0]


def work(case):
    """Fields read and written once by each solve (c and k in, c out) and each reaction, and the
    transforms of one D apply per PCG iteration, at two iterations a solve."""
    real = 8 if case["precision"] == "fp64" else 4

    def one(op, n, nt, gaussians):
        voxels = n ** 3
        fft = 2.5 * voxels * math.log2(voxels)
        if op == "smooth":
            return 2 * voxels * real, 2 * fft
        if op == "apply_d":
            return 3 * voxels * real, 6 * fft
        solves = {"diffusion": 1, "forward": 2 * nt}.get(op, 4 * nt)
        box = min(n, 2 * int(5 * max(SIGMA, 2 * math.pi / n) * n / (2 * math.pi)) + 1) ** 3
        return (solves * 4.5 * voxels + 2 * gaussians * box) * real, solves * 20 * fft

    if case["op"] != "batch":
        b, f = one(case["op"], case["n"], case["nt"], case["gaussians"])
    else:
        parts = [one("gradient", n, c["nt"], c["gaussians"])
                 for c, n, _ in batch_problems(case, 0)]
        b, f = (sum(v) for v in zip(*parts))
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits, with torch alone ----------------------------------------------------

class Exact:
    """The model in float64: spectral derivatives (Nyquist modes zeroed), PCG with the constant
    coefficient preconditioner stopped at 1e-6 of the preconditioned right-hand side, logistic
    reaction, Strang splitting."""

    def __init__(self, p, kappa, rho):
        n = self.n = p["n"]
        self.k = kappa * (p["wm"] + GM * p["gm"])
        self.wm, self.gm, self.rho = p["wm"], p["gm"], rho * p["wm"]
        self.filter = ((p["wm"] > 0.1) | (p["gm"] > 0.1)).double()
        kbar = float(self.k.sum() / self.filter.sum())
        w = torch.fft.fftfreq(n, 1 / n, device="cuda", dtype=torch.float64)
        w[n // 2] = 0
        self.w = [w[:, None, None], w[None, :, None], w[None, None, : n // 2 + 1]]
        w2 = sum(v * v for v in self.w)
        self.pc = 1 / (1 + 0.25 * (DT / 2) * kbar * w2)
        self.mult = torch.full((n // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
        self.mult[0] = self.mult[-1] = 1.0

    def back(self, s):
        return torch.fft.irfftn(s, s=(self.n,) * 3)

    def grad(self, s):
        return [self.back(1j * w * s) for w in self.w]

    def d_spec(self, s):
        out = 0
        for w in self.w:
            out = out + 1j * w * torch.fft.rfftn(self.k * self.back(1j * w * s))
        return out

    def dot(self, a, b):
        return float(((a.real * b.real + a.imag * b.imag) * self.mult).sum()) / self.n ** 3

    def diffuse(self, c, dt):
        a = 0.5 * dt
        x = torch.fft.rfftn(c)
        d = self.d_spec(x)
        b, r = x + a * d, 2 * a * d
        tol = 1e-6 * math.sqrt(self.dot(self.pc * b, self.pc * b))
        z = self.pc * r
        if math.sqrt(self.dot(z, z)) <= tol:
            return c
        beta, q = self.dot(z, r), z
        for _ in range(5000):
            v = q - a * self.d_spec(q)
            alpha = beta / self.dot(q, v)
            x = x + alpha * q
            r = r - alpha * v
            z = self.pc * r
            if math.sqrt(self.dot(z, z)) <= tol:
                break
            beta, old = self.dot(z, r), beta
            q = z + (beta / old) * q
        return self.back(x)

    def step(self, c):
        half = self.diffuse(c, DT / 2)
        e = half * torch.exp(self.rho * DT)
        return half, self.diffuse(e / (e + 1 - half), DT / 2)

    def linear_step(self, a, at):
        """The adjoint step around the half-step state (or the tangent step around c_i)."""
        a = self.diffuse(a, DT / 2)
        e = torch.exp(self.rho * DT)
        return self.diffuse(a * e / (at * e + 1 - at) ** 2, DT / 2)

    def basis(self, centers, sigma):
        """Each basis function on its box: ((slices), values), before normalisation."""
        n, x = self.n, axis(self.n)
        w = weierstrass(n, 2 * math.pi / n)
        for c in centers:
            far = [x - float(v) for v in c]
            g = [torch.exp(-(d / sigma) ** 2 / 2) for d in far]
            at = [torch.nonzero(d.abs() <= 5 * sigma).reshape(-1) for d in far]
            box = tuple(slice(int(i[0]), int(i[-1]) + 1) for i in at)
            f = self.filter * (g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :])
            v = along_axes(f, *(w[b] for b in box))
            r2 = sum((d[b] ** 2).reshape([-1 if k == j else 1 for k in range(3)])
                     for j, (d, b) in enumerate(zip(far, box)))
            yield box, torch.where(r2 <= 25 * sigma * sigma, v, torch.zeros_like(v))

    def phi(self, basis, coef):
        out, active = torch.zeros_like(self.k), [i for i, v in enumerate(coef) if v != 0]
        top = max(float(basis[i][1].max()) for i in active) if active else 1.0
        for i in active:
            out[basis[i][0]] += float(coef[i]) * basis[i][1]
        return out / top

    def phi_t(self, basis, v):
        top = max(float(f.max()) for _, f in basis)
        return np.array([float((f * v[box]).sum()) for box, f in basis]) / top


def exact_gradient(p, case, want_hessian=False):
    x = p["x"].astype(np.float64)
    m = Exact(p, float(x[-2]), float(x[-1]))
    basis = list(m.basis(p["centers"], p["sigma"]))
    h3 = (2 * math.pi / m.n) ** 3
    states, halves = [m.phi(basis, x[:-2])], []
    for _ in range(case["nt"]):
        half, c = m.step(states[-1])
        halves.append(half)
        states.append(c)
    if want_hessian:
        v = m.phi(basis, p["direction"][:-2])
        for c in states[:-1]:
            v = m.linear_step(v, c)
        a = -v
        for half in reversed(halves):
            a = m.linear_step(a, half)
        return np.concatenate([-h3 * m.phi_t(basis, a), [0.0, 0.0]])
    a = -(states[-1] - p["d1"].double())
    J = 0.5 * h3 * float((a * a).sum())
    dk = dr = 0.0
    for i in range(case["nt"], -1, -1):
        c, weight = states[i], (0.5 if i in (0, case["nt"]) else 1.0) * DT
        dots = sum(u * v for u, v in zip(m.grad(torch.fft.rfftn(c)), m.grad(torch.fft.rfftn(a))))
        dk += weight * float(((m.wm + GM * m.gm) * dots).sum())
        dr += weight * float((m.wm * (c * c - c) * a).sum())
        if i:
            a = m.linear_step(a, halves[i - 1])
    return (torch.tensor(J, dtype=torch.float64),
            np.concatenate([-h3 * m.phi_t(basis, a), [h3 * dk, h3 * dr]]))


def exact(case, seed):
    if case["op"] == "batch":
        return [exact_gradient(inputs(c, s, n), c) for c, n, s in batch_problems(case, seed)]
    p = inputs(case, seed, case["n"])
    if case["op"] in ("gradient", "hessian"):
        if case["precision"] == "fp64" and case["n"] >= 200:
            return None
        return exact_gradient(p, case, case["op"] == "hessian")
    m = Exact(p, case["kappa"], case["rho"])
    c, flat = p["c0"].double(), case["op"] in ("apply_d", "smooth", "diffusion")
    if case["op"] == "apply_d":
        out = m.back(m.d_spec(torch.fft.rfftn(c)))
    elif case["op"] == "smooth":
        out = smoothed(p["g"].double(), 2 * 2 * math.pi / m.n)
    elif case["op"] == "diffusion":
        out = m.diffuse(c, DT / 2)
    else:
        halves = []
        for _ in range(case["nt"]):
            half, c = m.step(c)
            halves.append(half)
        out = c
        if case["op"] == "adjoint":
            a = p["g"].double()
            for half in reversed(halves):
                a = m.linear_step(a, half)
            out = (c, a)
    return out.reshape(-1) if flat else out
