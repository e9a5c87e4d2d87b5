"""The calls a user of cfdfs makes, as measurable cases.

The library is a time-stepping solver with a C ABI and a Python binding, so
most cases are whole calls: time steps from a state in host memory to a state
in host memory, at the sizes and options of the test configurations and the
benchmark.  The others are the entry points that programs call by themselves:
the pressure solve, the solve on a caller's own device matrix, and the
network's forward pass, gradient and training step.

Kinds of case
  run      ``set_state``, ``run(steps)``, ``state``: what a driver does between
           two outputs.  The state is a small divergence-free flow that vanishes
           at the walls (cavity) or the impulsive start behind a parabolic inlet
           (duct), drawn from the seed.
  startup  ``Solver``, ``load``, ``step0`` and the first time step: a new deck.
  solve    ``pressure_solve`` of a caller's right-hand side, to the tolerance
           the training data of the network is made with.
  noalloc  ``pcg_solve_noalloc`` on a caller's CSR matrix in device memory.
  forward  the network's correction of one residual in device memory.
  gradient ``UNet.gradient`` of one host sample: loss and parameter gradients.
  train    ``UNet.train_batch`` on device samples: loss and updated parameters.
"""
import functools
import math
import os
import sys
import tempfile

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "cfd-with-cuda_b200"))

import cfdfs  # noqa: E402
from cfdfs import meshgen  # noqa: E402

WEIGHTS = os.path.join(_ROOT, "cfd-with-cuda_b200", "weights", "unet_cavity.bin")

# channels and grid level of the network's tensors, its convolutions (input
# tensor, output tensor, stride, leaky ReLU) and its two prolongation joins
# (coarse tensor, skip tensor, output tensor), in execution order
_T = [(0, 1), (0, 16), (1, 32), (1, 32), (2, 64), (2, 64), (2, 64), (2, 32), (1, 32), (1, 32), (1, 16), (0, 16),
      (0, 16), (0, 1)]
_NET = [("c", 0, 1, 1, 1), ("c", 1, 2, 2, 1), ("c", 2, 3, 1, 1), ("c", 3, 4, 2, 1), ("c", 4, 5, 1, 1),
        ("c", 5, 6, 1, 1), ("c", 6, 7, 1, 1), ("u", 7, 3, 8), ("c", 8, 9, 1, 1), ("c", 9, 10, 1, 1),
        ("u", 10, 1, 11), ("c", 11, 12, 1, 1), ("c", 12, 13, 1, 0)]


def listed():
    return [
        # the smallest configuration (8^3 cavity, Re 100): launches and waits
        dict(name="cavity8_fp64", kind="run", nx=8, ny=8, nz=8, re=100.0, dt=0.01, ngp=8, grading=0.0,
             method="fp64_jacobi", steps=4),
        # the mid-size FP64 configuration (32^3 cavity, Re 400)
        dict(name="cavity32_fp64", kind="run", nx=32, ny=32, nz=32, re=400.0, dt=0.005, ngp=8, grading=0.0,
             method="fp64_jacobi", steps=2),
        # the reference's algorithm at the benchmark's size (64^3 cavity, Re 1000)
        dict(name="cavity64_fp64", kind="run", nx=64, ny=64, nz=64, re=1000.0, dt=0.002, ngp=8, grading=0.0,
             method="fp64_jacobi", steps=1),
        # the fastest path at the benchmark's size
        dict(name="cavity64_twolevel", kind="run", nx=64, ny=64, nz=64, re=1000.0, dt=0.002, ngp=8, grading=0.0,
             method="mixed_twolevel", steps=3),
        # the benchmark's headline path: the network in the first iteration of a solve
        dict(name="cavity64_learned", kind="run", nx=64, ny=64, nz=64, re=1000.0, dt=0.002, ngp=8, grading=0.0,
             method="mixed_learned", steps=3),
        # the bent duct (24 x 24 x 160, parabolic inlet): non-cubic, non-affine
        dict(name="duct_learned", kind="run", nx=160, ny=24, nz=24, re=200.0, dt=0.005, ngp=8, grading=-1.0,
             method="mixed_learned", steps=3),
        # a new deck with 27 Gauss points on a graded 30^3 mesh, up to its first step
        dict(name="startup30_ngp27", kind="startup", nx=30, ny=30, nz=30, re=400.0, dt=0.002, ngp=27, grading=1.5,
             method="fp64_jacobi", steps=1),
        # the solve that makes the network's training data (FP64 two-level CG, 1e-12)
        dict(name="solve64_twolevel", kind="solve", nx=64, ny=64, nz=64, grading=0.0, method="fp64_twolevel",
             rtol=1e-12),
        # a coupled code's own 27-point operator, odd sizes, no device allocation
        dict(name="noalloc_65x63x61", kind="noalloc", nx=65, ny=63, nz=61, rtol=1e-8),
        # one application of the network on the benchmark's pressure grid
        dict(name="unet_forward65", kind="forward", nx=65, ny=65, nz=65),
        # one sample's gradient on the benchmark's pressure grid
        dict(name="unet_gradient65", kind="gradient", nx=65, ny=65, nz=65),
        # a fine-tuning step (batch 4) on the duct's pressure grid
        dict(name="unet_train_duct", kind="train", nx=161, ny=25, nz=25, batch=4, lr=1e-5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "startup", "solve", "noalloc", "forward", "gradient", "train"])
    if kind in ("run", "startup"):
        method = rng.choice(["fp64_jacobi", "mixed_jacobi", "mixed_twolevel", "mixed_learned"])
        if kind == "run" and rng.random() < 0.3:  # the bent duct
            c = 4 * _log_int(rng, 1, 6) if method == "mixed_learned" else _log_int(rng, 4, 24)
            a = 4 * _log_int(rng, 4, 40) if method == "mixed_learned" else _log_int(rng, 16, 160)
            return dict(kind=kind, nx=a, ny=c, nz=c, re=round(rng.uniform(100.0, 300.0), 1), dt=0.002, ngp=8,
                        grading=-1.0, method=method, steps=rng.randint(1, 2))
        hi = 30 if kind == "startup" else 60
        n = 4 * _log_int(rng, 2, hi // 4) if method == "mixed_learned" else _log_int(rng, 6, hi)
        re = round(rng.uniform(100.0, 1000.0), 1)
        # the scheme takes viscosity explicitly: nu dt / h^2 <= 0.08 at the finest spacing
        dt = float("%.3g" % min(0.01 if n <= 10 else 0.002, 0.08 * re * (0.35 / n) ** 2))
        return dict(kind=kind, nx=n, ny=n, nz=n, re=re, dt=dt, ngp=rng.choice([8, 8, 27]),
                    grading=rng.choice([0.0, 0.0, 1.0, 1.5]), method=method,
                    steps=1 if kind == "startup" else rng.randint(1, 2))
    if kind == "solve":
        n = _log_int(rng, 6, 60)
        method = rng.choice(["fp64_jacobi", "fp64_twolevel"])
        return dict(kind=kind, nx=n, ny=n, nz=n, grading=rng.choice([0.0, 1.5]), method=method,
                    rtol=1e-12 if method == "fp64_twolevel" else 1e-8)
    if kind == "noalloc":
        return dict(kind=kind, nx=_log_int(rng, 5, 64), ny=_log_int(rng, 5, 64), nz=_log_int(rng, 5, 61),
                    rtol=rng.choice([1e-6, 1e-8, 1e-10]))
    dims = [4 * _log_int(rng, 1, 16) + 1 for _ in range(3)]
    c = dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2])
    if kind == "train":
        c.update(batch=rng.randint(1, 4), lr=1e-5)
    return c


# ---- time steps and pressure solves ----------------------------------------

_METHODS = {
    # the reference's algorithm: FP64, Jacobi-PCG from x0 = 0
    "fp64_jacobi": dict(precision=cfdfs.FP64, precond=cfdfs.PC_JACOBI),
    "fp64_twolevel": dict(precision=cfdfs.FP64, precond=cfdfs.PC_TWOLEVEL, cg_maxit=20000),
    "mixed_jacobi": dict(precision=cfdfs.MIXED, precond=cfdfs.PC_JACOBI),
    # the benchmark's options: warm start, FP32 inner solves to 1e-5
    "mixed_twolevel": dict(precision=cfdfs.MIXED, precond=cfdfs.PC_TWOLEVEL, cg_warm=1, inner_rtol=1e-5),
    "mixed_learned": dict(precision=cfdfs.MIXED, precond=cfdfs.PC_LEARNED, cg_warm=1, inner_rtol=1e-5,
                          fcg_net_iters=1),
}


@functools.lru_cache(maxsize=3)
def _deck_text(nx, ny, grading, re, dt, ngp):
    if grading < 0:
        return meshgen.duct_deck(n_cross=ny, n_axial=nx, re=re, dt=dt, steps=100, ngp=ngp)
    return meshgen.cavity_deck(meshgen.CavitySpec(nx, re=re, dt=dt, steps=100, ngp=ngp, grading=grading))


class _Deck:
    """A deck file that is removed with the object."""

    def __init__(self, case):
        fd, self.path = tempfile.mkstemp(suffix=".inp")
        with os.fdopen(fd, "w") as f:
            f.write(_deck_text(case["nx"], case["ny"], case["grading"], case.get("re", 100.0), case.get("dt", 0.01),
                               case.get("ngp", 8)))

    def remove(self):
        if self.path:
            os.unlink(self.path)
            self.path = None

    __del__ = remove


@functools.lru_cache(maxsize=3)
def _geometry(nx, ny, nz, grading):
    """Velocity-node coordinates (NN x 3) and, for the duct, its inlet profile."""
    d = _Deck(dict(nx=nx, ny=ny, nz=nz, grading=grading))
    m = cfdfs.HostMesh(d.path)
    xyz = m.coord()
    inlet = meshgen.duct_inlet_profile(m) if grading < 0 else None
    m.close()
    d.remove()
    return xyz, inlet


def _vortices(xyz, seed):
    """Three random vortex sheets, divergence-free and zero on the walls of
    the unit cube: [u | v | w]."""
    rng = np.random.default_rng(seed)
    x = torch.from_numpy(xyz.T.copy()).cuda()
    u = torch.zeros_like(x)
    for a, b in ((0, 1), (1, 2), (2, 0)):
        for _ in range(2):
            m = [int(k) for k in rng.integers(1, 3, size=3)]
            amp = 0.06 * float(rng.uniform(-1.0, 1.0))
            s = [torch.sin(m[k] * math.pi * x[k]) ** 2 for k in range(3)]
            ds = [m[k] * math.pi * torch.sin(2 * m[k] * math.pi * x[k]) for k in range(3)]
            c = 3 - a - b
            u[a] += amp * s[a] * ds[b] * s[c]
            u[b] -= amp * ds[a] * s[b] * s[c]
    return u.reshape(-1).cpu().numpy()


def _new_solver(case, path):
    s = cfdfs.Solver(device=0, **_METHODS[case["method"]])
    s.load(path)
    s.step0()
    if case["grading"] < 0:
        s.set_pressure_grid(meshgen.duct_grid_dims(case["ny"], case["nx"]))
    if case["method"] == "mixed_learned":
        s.load_unet(WEIGHTS, (case["nx"] + 1, case["ny"] + 1, case["nz"] + 1))
    return s


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _prepare_run(case, seed):
    deck = _Deck(case)
    xyz, inlet = _geometry(case["nx"], case["ny"], case["nz"], case["grading"])
    s = _new_solver(case, deck.path)
    if case["method"] in ("mixed_twolevel", "mixed_learned"):
        s.precond_apply(np.zeros(s.info.NNp))  # builds the coarse space before the first step
    if inlet is not None:
        peak = float(np.random.default_rng(seed).uniform(0.7, 1.3))
        s.set_bc_values(inlet[0], peak * inlet[1])
    u0, p0 = _pinned(3 * s.info.NN), _pinned(s.info.NNp)
    s.state(out=(u0, p0))
    if inlet is None:
        u0 += _vortices(xyz, seed)
    return dict(case=case, solver=s, start=(u0, p0), out=(_pinned(u0.size), _pinned(p0.size)))


def _run_run(st):
    s = st["solver"]
    s.set_state(*st["start"])
    s.run(st["case"]["steps"])
    u, p = s.state(out=st["out"])
    return {"u": u, "p": p}


def _prepare_startup(case, seed):
    xyz, _ = _geometry(case["nx"], case["ny"], case["nz"], case["grading"])
    return dict(case=case, deck=_Deck(case), flow=_vortices(xyz, seed))


def _run_startup(st):
    s = _new_solver(st["case"], st["deck"].path)
    u, p = s.state()
    s.set_state(u + st["flow"], p)
    s.run(st["case"]["steps"])
    u, p = s.state()
    s.close()
    return {"u": u, "p": p}


def _prepare_solve(case, seed):
    deck = _Deck(case)
    s = cfdfs.Solver(device=0, cg_rtol=case["rtol"], **{"cg_maxit": 20000, **_METHODS[case["method"]]})
    s.load(deck.path)
    s.step0()
    if case["method"] == "fp64_twolevel":
        s.precond_apply(np.zeros(s.info.NNp))
    m = case["nx"] + 1
    rhs = _field(m, m, m, seed).double().cpu().numpy().reshape(-1)
    return dict(case=case, solver=s, rhs=rhs)


def _run_solve(st):
    x, _ = st["solver"].pressure_solve(st["rhs"])
    return {"x": x}


# ---- the solve on a caller's matrix ------------------------------------------

def _axis_terms(n):
    """1D linear-element mass and stiffness bands (lower, diagonal, upper) on
    n nodes with unit spacing and natural ends."""
    k = torch.full((n, 3), -1.0, dtype=torch.float64)
    m = torch.full((n, 3), 1.0 / 6.0, dtype=torch.float64)
    k[:, 1], m[:, 1] = 2.0, 4.0 / 6.0
    for i in (0, n - 1):
        k[i, 1], m[i, 1] = 1.0, 2.0 / 6.0
    k[0, 0] = k[n - 1, 2] = m[0, 0] = m[n - 1, 2] = 0.0
    return k.cuda(), m.cuda()


def _taps27(nx, ny, nz):
    """Trilinear-element Laplacian plus a small mass term, as 27 coefficients
    per node: (27, nz, ny, nx), tap dx fastest."""
    (kx, mx), (ky, my), (kz, mz) = _axis_terms(nx), _axis_terms(ny), _axis_terms(nz)
    taps = []
    for t in range(27):
        a, b, c = t % 3, (t // 3) % 3, t // 9
        X = lambda v: v[:, a][None, None, :]  # noqa: E731
        Y = lambda v: v[:, b][None, :, None]  # noqa: E731
        Z = lambda v: v[:, c][:, None, None]  # noqa: E731
        taps.append(X(kx) * Y(my) * Z(mz) + X(mx) * Y(ky) * Z(mz) + X(mx) * Y(my) * Z(kz) +
                    1e-3 * X(mx) * Y(my) * Z(mz))
    return torch.stack([t.expand(nz, ny, nx) for t in taps])


def _apply27(taps, x):
    nz, ny, nx = x.shape
    p = torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))
    y = torch.zeros_like(x)
    for t in range(27):
        a, b, c = t % 3, (t // 3) % 3, t // 9
        y += taps[t] * p[c:c + nz, b:b + ny, a:a + nx]
    return y


def _field(nx, ny, nz, seed):
    """A residual-like field (nz, ny, nx), FP32, unit RMS: low modes plus
    grid-scale noise."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    r = np.random.default_rng(seed)
    ax = [torch.linspace(0.0, math.pi, n, device="cuda") for n in (nx, ny, nz)]
    f = 0.3 * torch.randn(nz, ny, nx, device="cuda", generator=g)
    for _ in range(6):
        k = r.integers(0, 5, size=3)
        f += float(r.normal()) * (torch.cos(int(k[2]) * ax[2])[:, None, None] *
                                  torch.cos(int(k[1]) * ax[1])[None, :, None] *
                                  torch.cos(int(k[0]) * ax[0] + 0.3)[None, None, :])
    return f / f.square().mean().sqrt()


def _prepare_noalloc(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    taps = _taps27(nx, ny, nz)
    z, y, x = torch.meshgrid(torch.arange(nz), torch.arange(ny), torch.arange(nx), indexing="ij")
    cols, keep = [], []
    for t in range(27):
        a, b, c = x + t % 3 - 1, y + (t // 3) % 3 - 1, z + t // 9 - 1
        keep.append((a >= 0) & (a < nx) & (b >= 0) & (b < ny) & (c >= 0) & (c < nz))
        cols.append(a + nx * (b + ny * c))
    keep = torch.stack(keep, -1).reshape(-1, 27).cuda()
    cols = torch.stack(cols, -1).reshape(-1, 27).cuda()
    vals = taps.permute(1, 2, 3, 0).reshape(-1, 27)
    rowptr = torch.zeros(nx * ny * nz + 1, dtype=torch.int32, device="cuda")
    rowptr[1:] = keep.sum(1).cumsum(0).to(torch.int32)
    return dict(case=case, n=nx * ny * nz, rowptr=rowptr, col=cols[keep].to(torch.int32).contiguous(),
                val=vals[keep].contiguous(), dinv=(1.0 / taps[13]).reshape(-1).contiguous(),
                b=_field(nx, ny, nz, seed).double().reshape(-1).contiguous(),
                x=torch.zeros(nx * ny * nz, dtype=torch.float64, device="cuda"))


def _run_noalloc(st):
    rc, _, msg = cfdfs.pcg_solve_noalloc(st["rowptr"].data_ptr(), st["col"].data_ptr(), st["val"].data_ptr(),
                                         st["dinv"].data_ptr(), st["b"].data_ptr(), st["x"].data_ptr(), st["n"],
                                         st["case"]["rtol"], 2000, torch.cuda.current_stream().cuda_stream)
    if rc != cfdfs.CFD_OK:
        raise RuntimeError(msg)
    return {"x": st["x"]}


def _exact_noalloc(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    taps = _taps27(nx, ny, nz)
    b = _field(nx, ny, nz, seed).double()
    x, r = torch.zeros_like(b), b.clone()
    z = r / taps[13]
    p, rz, stop = z.clone(), (r * z).sum(), 1e-13 * b.norm()
    for _ in range(2000):
        q = _apply27(taps, p)
        al = rz / (p * q).sum()
        x += al * p
        r -= al * q
        if r.norm() <= stop:
            break
        z = r / taps[13]
        new = (r * z).sum()
        p = z + new / rz * p
        rz = new
    return {"x": x.reshape(-1)}


# ---- the network ---------------------------------------------------------------

def _dims(case):
    return (case["nx"], case["ny"], case["nz"])


def _prepare_net(case, seed):
    net = cfdfs.UNet(device=0, path=WEIGHTS)
    nb = case.get("batch", 1)
    x = torch.stack([_field(*_dims(case), 2 * seed + 1000 * i) for i in range(nb)])
    t = torch.stack([0.3 * _field(*_dims(case), 2 * seed + 1000 * i + 1) for i in range(nb)])
    st = dict(case=case, net=net, x=x.contiguous(), t=t.contiguous(), y=torch.zeros_like(x[0]))
    if case["kind"] == "gradient":
        st["x"], st["t"] = x[0].cpu().numpy(), t[0].cpu().numpy()
    return st


def _run_net(st):
    case, net = st["case"], st["net"]
    if case["kind"] == "forward":
        net.forward_device(st["x"].data_ptr(), st["y"].data_ptr(), _dims(case))
        return {"y": st["y"]}
    if case["kind"] == "gradient":
        loss, grad = net.gradient(st["x"], st["t"])
        return {"loss": np.float32(loss), "grad": grad}
    loss = net.train_batch(st["x"].data_ptr(), st["t"].data_ptr(), _dims(case), case["lr"], on_device=True,
                           nb=case["batch"])
    return {"loss": np.float32(loss), "params": net.params()}


class _Stored(torch.autograd.Function):
    """A BF16-stored value: rounded forward, passed through backward."""

    @staticmethod
    def forward(ctx, v):
        return v.float().bfloat16().double()

    @staticmethod
    def backward(ctx, g):
        return g


def _up(v):
    """Vertex-centred trilinear prolongation of (Z, Y, X, C)."""
    for ax in range(3):
        n = v.shape[ax]
        lo, hi = v.narrow(ax, 0, n - 1), v.narrow(ax, 1, n - 1)
        mid = torch.stack([lo, 0.5 * (lo + hi)], dim=ax + 1).flatten(ax, ax + 1)
        v = torch.cat([mid, v.narrow(ax, n - 1, 1)], dim=ax)
    return v


def _net64(theta, x):
    """The network in 64 bits, with weights and stored activations rounded to
    BF16 where it stores them so."""
    acts, o = {0: _Stored.apply(x.double()[..., None])}, 0
    for op in _NET:
        if op[0] == "u":
            acts[op[3]] = _Stored.apply(_up(acts[op[1]]) + acts[op[2]])
            continue
        _, ti, to, stride, act = op
        cin, cout = _T[ti][1], _T[to][1]
        w = _Stored.apply(theta[o:o + 27 * cin * cout]).reshape(27, cin, cout)
        y = theta[o + 27 * cin * cout:o + 27 * cin * cout + cout]
        o += 27 * cin * cout + cout
        v = acts[ti]
        shape = [(n - 1) // stride + 1 for n in v.shape[:3]]
        p = torch.nn.functional.pad(v, (0, 0, 1, 1, 1, 1, 1, 1))
        for k in range(27):
            d = (k // 9, (k // 3) % 3, k % 3)
            win = p[tuple(slice(d[i], d[i] + stride * (shape[i] - 1) + 1, stride) for i in range(3))]
            y = y + win @ w[k]
        if act:
            y = torch.where(y < 0, 0.1 * y, y)
        acts[to] = y if to == len(_T) - 1 else _Stored.apply(y)
    return acts[len(_T) - 1][..., 0]


def _exact_net(case, seed):
    st = _prepare_net(case, seed)
    theta = torch.from_numpy(st["net"].params().astype(np.float64)).cuda()
    st["net"].close()
    if case["kind"] == "forward":
        with torch.no_grad():
            return {"y": _net64(theta, st["x"][0])}
    nb = case.get("batch", 1)
    x, t = torch.as_tensor(st["x"]).cuda(), torch.as_tensor(st["t"]).cuda()
    x, t = x.reshape(nb, *x.shape[-3:]), t.reshape(nb, *t.shape[-3:])
    grad, loss = torch.zeros_like(theta), 0.0
    for i in range(nb):
        p = theta.clone().requires_grad_(True)
        li = (_net64(p, x[i]) - t[i].double()).square().mean()
        li.backward()
        grad += p.grad / nb
        loss += float(li) / nb
    if case["kind"] == "gradient":
        return {"loss": loss, "grad": grad}
    # the first Adam step: both moments' bias corrections leave g / (|g| + eps)
    return {"loss": loss, "params": theta - case["lr"] * grad / (grad.abs() + 1e-8)}


# ---- the interface -----------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "run":
        return _prepare_run(case, seed)
    if kind == "startup":
        return _prepare_startup(case, seed)
    if kind == "solve":
        return _prepare_solve(case, seed)
    if kind == "noalloc":
        return _prepare_noalloc(case, seed)
    return _prepare_net(case, seed)


def run(state):
    kind = state["case"]["kind"]
    if kind == "run":
        return _run_run(state)
    if kind == "startup":
        return _run_startup(state)
    if kind == "solve":
        return _run_solve(state)
    if kind == "noalloc":
        return _run_noalloc(state)
    return _run_net(state)


def exact(case, seed):
    # time steps and the solver's own pressure operator have no value without
    # the solver's assembly
    if case["kind"] == "noalloc":
        return _exact_noalloc(case, seed)
    if case["kind"] in ("forward", "gradient", "train"):
        return _exact_net(case, seed)
    return None


def _net_work(nx, ny, nz):
    """Multiply-adds x 2 and stored bytes of one forward pass."""
    d = [(nx, ny, nz)]
    for _ in range(2):
        d.append(tuple((n - 1) // 2 + 1 for n in d[-1]))
    vox = [float(a[0] * a[1] * a[2]) for a in d]
    flops = sum(2.0 * 27 * _T[o[1]][1] * _T[o[2]][1] * vox[_T[o[2]][0]] for o in _NET if o[0] == "c")
    return flops, 8.0 * vox[0]


def work(case):
    kind, (nx, ny, nz) = case["kind"], _dims(case)
    if kind in ("forward", "gradient", "train"):
        flops, io = _net_work(nx, ny, nz)
        par = 4.0 * cfdfs.UNet.param_count()
        if kind == "forward":
            return {"bytes": io + par / 2, "flops": flops}
        nb = case.get("batch", 1)  # backward: twice the forward's products
        return {"bytes": nb * io + (2 if kind == "gradient" else 8) * par, "flops": 3.0 * nb * flops}
    if kind == "noalloc":
        n = nx * ny * nz
        its = 1.5 * max(nx, ny, nz)  # Jacobi-PCG on a grid: proportional to its longest side
        nnz = (3.0 * nx - 2) * (3.0 * ny - 2) * (3.0 * nz - 2)
        return {"bytes": its * (12.0 * nnz + 4.0 * n + 8.0 * 10 * n), "flops": its * (2.0 * nnz + 12.0 * n)}
    # non-zeros: Z couples corner nodes within two steps per axis, K (hex27)
    # has about 63 and G about 15.4 entries per velocity node
    npr, nv = (nx + 1.0) * (ny + 1.0) * (nz + 1.0), (2.0 * nx + 1) * (2.0 * ny + 1) * (2.0 * nz + 1)
    nnz_z, nnz_k, nnz_g = npr * 117.0, nv * 63.0, nv * 15.4
    mixed = case["method"].startswith("mixed")
    s = 4.0 if mixed else 8.0
    # Krylov iterations per solve: Jacobi-PCG about two per element along the
    # longest side, the two-level preconditioner about 25 whatever the size
    its = 2.0 * max(nx, ny, nz) if case["method"].endswith("jacobi") else 25.0
    solve_b, solve_f = its * (nnz_z * s + 9.0 * npr * s), its * (2.0 * nnz_z + 12.0 * npr)
    if kind == "solve":
        return {"bytes": 1.5 * solve_b, "flops": 1.5 * solve_f}
    sub = 3.0 * case["steps"]  # sub-iterations: about three per step from these states
    stage_b = (2.0 * nnz_k + 3.0 * 3.0 * nnz_g) * s + 30.0 * 3.0 * nv * s
    stage_f = 2.0 * 3.0 * (2.0 * nnz_k + 3.0 * nnz_g)
    b, f = sub * (solve_b + stage_b) + 8.0 * 2.0 * (3.0 * nv + npr), sub * (solve_f + stage_f)
    if kind == "startup":
        b += 8.0 * (nnz_k + 6.0 * nnz_g + nnz_z)
    return {"bytes": b, "flops": f}
