"""Performance cases: the work a user of this framework has it do, through its public entry points.

A case is a dict of plain values; ``kind`` says which path it takes:

  step      LLGIntegrator.step: adaptive Runge-Kutta steps of one film or block (hmax bounds the step)
  field     one field evaluation of a device-resident magnetisation, and (``energy``) the total energy
  tensor    DemagField(mesh): assembly of the demagnetisation tensor of a new mesh
  minimize  LBFGS_Minimizer.minimize from a given magnetisation
  ensemble  StochasticBatch.steps: Langevin members of uneven sizes advanced together
  train     UNet.train_step of the learned warm start (forward, backward, Adam)
  propose   UNet.forward: the warm start's proposal for a few films

``listed()`` holds the standing cases, ``draw(rng)`` makes more of the same ranges, ``prepare`` / ``run`` execute one,
``work`` counts what a pass cannot do without and ``exact`` gives the outputs in plain 64-bit torch arithmetic.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "magnum.af_b200", "python"))

import magnumaf as M  # noqa: E402
from magnumaf.unet import UNet  # noqa: E402

MU0 = 4e-7 * math.pi
GAMMA = 1.760859644e11 * MU0
KB = 1.38064852e-23

# materials: name -> cell, Ms, exchange A, interface DMI D (axis z), uniaxial Ku (axis z), cubic K1 (axes x, y, z),
# uniform field H, damping
MATERIALS = {
    "permalloy": dict(cell=(5e-9, 5e-9, 3e-9), Ms=8e5, A=1.3e-11, alpha=0.02),
    "cobalt_film": dict(cell=(2e-9, 2e-9, 1e-9), Ms=1.1e6, A=1.6e-11, D=3e-3, Ku=1e6, alpha=0.1),
    "iron_block": dict(cell=(3e-9, 3e-9, 3e-9), Ms=8.6e5, A=1.3e-11, K1=-1e4, H=(2e4, -1.1e4, 8e3), alpha=0.01),
}


def listed():
    return [
        # the muMAG standard problem 4 strip: the smallest simulation everybody runs first
        dict(name="strip_step_fp64", kind="step", nx=100, ny=25, nz=1, material="permalloy", precision="fp64",
             scheme="DP45", geometry="box", start="smooth", steps=1),
        # a thin film of decimal size, interface DMI and anisotropy
        dict(name="film_step_fp64", kind="step", nx=300, ny=200, nz=1, material="cobalt_film", precision="fp64",
             scheme="RKF45", geometry="box", start="smooth", steps=1),
        # the skyrmion film
        dict(name="skyrmion_step_fp32", kind="step", nx=512, ny=512, nz=4, material="cobalt_film",
             precision="fp32_field", scheme="RKF45", geometry="box", start="discs", steps=1),
        # a patterned disc: cells outside it are empty, so the state carries a field of Ms
        dict(name="disc_step_fp32", kind="step", nx=180, ny=180, nz=9, material="permalloy", precision="fp32_field",
             scheme="RKF45", geometry="disc", start="smooth", steps=1),
        # a thick block in double precision, random start
        dict(name="block_step_fp64", kind="step", nx=512, ny=512, nz=16, material="iron_block", precision="fp64",
             scheme="DP45", geometry="box", start="random", steps=1),
        # the benchmark's field evaluation: the largest mesh
        dict(name="block_field_fp32", kind="field", nx=1024, ny=1024, nz=16, material="iron_block",
             precision="fp32_field", start="random", energy=False),
        # field and energy of a bar of odd sizes, as monitored while relaxing
        dict(name="bar_field_energy_fp64", kind="field", nx=125, ny=75, nz=40, material="iron_block",
             precision="fp64", start="smooth", energy=True),
        # a new mesh: every program that uses the demagnetising field begins with this
        dict(name="tensor_assembly", kind="tensor", nx=200, ny=120, nz=10, material="permalloy"),
        # energy minimisation of a film, twenty iterations
        dict(name="film_minimize_fp64", kind="minimize", nx=128, ny=128, nz=1, material="cobalt_film",
             precision="fp64", demag=True, iterations=20),
        # Langevin ensemble of square and oblong films
        dict(name="ensemble_heun_fp32", kind="ensemble", members=16, max_side=512, steps=10),
        # one training step of the warm-start network
        dict(name="unet_train_bf16", kind="train", B=16, H=128, W=128),
        # its proposal for one film: latency
        dict(name="unet_propose_bf16", kind="propose", B=1, H=128, W=128),
    ]


def _smooth(n):
    """Whether n has no prime factor above 13 (the lengths the transforms support)."""
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def _size(rng, lo, hi):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    while not _smooth(v):
        v -= 1
    return max(v, lo if _smooth(lo) else 1)


def draw(rng):
    kind = rng.choice(["step", "step", "step", "field", "field", "tensor", "minimize", "ensemble", "train", "propose"])
    material = rng.choice(sorted(MATERIALS))
    precision = rng.choice(["fp64", "fp32_field"])
    scheme = rng.choice(["RKF45", "DP45", "BS23"])
    if kind == "step":
        if rng.random() < 0.5:
            nx, ny, nz = _size(rng, 24, 900), _size(rng, 16, 900), 1
        else:
            nx, ny, nz = _size(rng, 32, 512), _size(rng, 32, 512), _size(rng, 2, 16)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, material=material, precision=precision, scheme=scheme,
                    geometry=rng.choice(["box", "box", "disc"]), start=rng.choice(["smooth", "discs", "random"]), steps=1)
    if kind == "field":
        return dict(kind=kind, nx=_size(rng, 32, 1024), ny=_size(rng, 32, 1024), nz=_size(rng, 1, 16),
                    material=material, precision=precision, start=rng.choice(["smooth", "random"]),
                    energy=rng.random() < 0.5)
    if kind == "tensor":
        return dict(kind=kind, nx=_size(rng, 24, 300), ny=_size(rng, 24, 300), nz=_size(rng, 1, 12), material=material)
    if kind == "minimize":
        return dict(kind=kind, nx=_size(rng, 64, 256), ny=_size(rng, 64, 256), nz=1, material="cobalt_film",
                    precision="fp64", demag=rng.random() < 0.5, iterations=rng.randint(10, 20))
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(4, 24), max_side=rng.choice([128, 256, 512]),
                    steps=2 * rng.randint(2, 6))
    return dict(kind=kind, B=rng.randint(2, 16) if kind == "train" else rng.randint(1, 8),
                H=16 * rng.randint(4, 8), W=16 * rng.randint(4, 8))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(seed, n):
    return np.random.default_rng(int(seed)).uniform(size=n)


def magnetisation(case, seed):
    """Unit vectors [3][nz][ny][nx] in FP64 on the GPU (zero outside a disc)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    start = case.get("start", "smooth")
    if start == "random":
        m = torch.randn((3, nz, ny, nx), generator=_gen(seed), dtype=torch.float64, device="cuda")
    else:
        x = torch.arange(nx, dtype=torch.float64, device="cuda")[None, None, :]
        y = torch.arange(ny, dtype=torch.float64, device="cuda")[None, :, None]
        z = torch.arange(nz, dtype=torch.float64, device="cuda")[:, None, None]
        u = _uniform(seed, 512)
        if start == "smooth":  # a few low Fourier modes per component
            m = torch.zeros((3, nz, ny, nx), dtype=torch.float64, device="cuda")
            i = 0
            for c in range(3):
                m[c] = 0.3 + u[500 + c]
                for kx in range(4):
                    for ky in range(4):
                        a, b = (2 * u[i] - 1) / (1 + kx + ky), 2 * math.pi * u[i + 1]
                        m[c] += a * torch.cos(math.pi * (kx * x / nx + ky * y / ny + 0.5 * z / nz) + b)
                        i += 2
        else:  # up, with reversed discs (skyrmion seeds)
            mz = torch.ones((nz, ny, nx), dtype=torch.float64, device="cuda")
            for k in range(20):
                r = 5 + 10 * u[3 * k]
                d2 = (x - nx * u[3 * k + 1]) ** 2 + (y - ny * u[3 * k + 2]) ** 2
                mz = torch.where((d2 <= r * r).expand(nz, ny, nx), -torch.ones_like(mz), mz)
            m = torch.stack([torch.zeros_like(mz), torch.zeros_like(mz), mz])
            m = m + 0.02 * torch.randn(m.shape, generator=_gen(seed), dtype=torch.float64, device="cuda")
    m /= m.square().sum(0, keepdim=True).sqrt()
    if case.get("geometry") == "disc":
        x = (torch.arange(nx, dtype=torch.float64, device="cuda")[None, None, :] + 0.5) / nx - 0.5
        y = (torch.arange(ny, dtype=torch.float64, device="cuda")[None, :, None] + 0.5) / ny - 0.5
        m = m * (x * x + y * y <= 0.25).to(torch.float64)
    return m.contiguous()


def _host(m):
    """(nx, ny, nz, 3) NumPy view, Fortran order, of a device field [3][nz][ny][nx]."""
    return m.cpu().numpy().transpose(3, 2, 1, 0)


def _terms(mesh, mat, demag=True):
    t = [M.DemagField(mesh)] if demag else []
    t.append(M.ExchangeField(mat["A"]))
    if "D" in mat:
        t.append(M.DmiField(mat["D"]))
    if "Ku" in mat:
        t.append(M.UniaxialAnisotropyField(mat["Ku"]))
    if "K1" in mat:
        t.append(M.CubicAnisotropyField(mat["K1"]))
    if "H" in mat:
        t.append(M.ExternalField.uniform(*mat["H"]))
    return t


def _step_size(case):
    """The bound on the time step (s): well inside the error tolerance, so that every step takes it."""
    return (2e-14 if case["start"] == "smooth" else 6e-15) * (0.1 if case["scheme"] == "BS23" else 1.0)


class _DeviceM:
    """The state's own device buffer as an array; holds the state, whose buffer goes with it."""

    def __init__(self, state):
        md = state.mesh
        self.state = state
        self.__cuda_array_interface__ = dict(shape=(3, md.nz, md.ny, md.nx), typestr="<f8",
                                             data=(state.device_m(), False), version=3)


def _device_m(state):
    return torch.as_tensor(_DeviceM(state), device="cuda")


SIDES = [64, 96, 128, 192, 256, 384, 512]


def _members(case, seed):
    """(nx, ny) of every member; the sizes belong to the case, not to the seed."""
    rng = np.random.default_rng(case["members"])
    sides = [s for s in SIDES if s <= case["max_side"]]
    return [(int(rng.choice(sides)), int(rng.choice(sides))) for _ in range(case["members"])]


def _unet_inputs(case, seed):
    B, H, W = case["B"], case["H"], case["W"]
    g = _gen(seed)
    x = torch.randn((B, 8, H, W), generator=g, dtype=torch.float32, device="cuda")
    x[:, :3] /= x[:, :3].square().sum(1, keepdim=True).sqrt()
    x[:, 3:] = torch.rand((B, 5, 1, 1), generator=g, dtype=torch.float32, device="cuda") * 2
    # targets: relaxed films vary slowly
    k = torch.arange(3, dtype=torch.float32, device="cuda")
    cx = torch.cos(math.pi * k[:, None] * torch.arange(W, dtype=torch.float32, device="cuda") / W)
    cy = torch.cos(math.pi * k[:, None] * torch.arange(H, dtype=torch.float32, device="cuda") / H)
    a = torch.randn((B, 3, 3, 3), generator=g, dtype=torch.float32, device="cuda")
    a[..., 0, 0] += torch.tensor([0.5, -0.5, 1.5], device="cuda")
    t = (cy.t() @ (a @ cx)).permute(0, 2, 3, 1)
    t = t / t.square().sum(3, keepdim=True).sqrt()
    return x.contiguous(), t.reshape(-1, 3).contiguous()


def _unet_params(net, seed):
    """He-initialised weights, small biases and a last layer that is not zero (a network in training)."""
    rng = np.random.default_rng(seed)
    p = net.get_params()
    for L in net.layers:
        p[L.boff:L.boff + L.cout] = rng.normal(0, 0.02, size=L.cout)
    L = net.layers[-1]
    p[L.woff:L.boff] = rng.normal(0, 0.03, size=L.boff - L.woff)
    return p


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("train", "propose"):
        net = UNet(8, seed=seed)
        net.set_params(_unet_params(net, seed))
        x, t = _unet_inputs(case, seed)
        return dict(case=case, net=net, x=x, t=t)
    if kind == "ensemble":
        mat = MATERIALS["cobalt_film"]
        members = []
        for i, (nx, ny) in enumerate(_members(case, seed)):
            mesh = M.Mesh(nx, ny, 1, *mat["cell"])
            m = magnetisation(dict(nx=nx, ny=ny, nz=1, start="smooth"), seed + 1000 * i)
            st = M.State(mesh, mat["Ms"], _host(m), precision="fp32_field")
            it = M.Stochastic_LLG(mat["alpha"], 300.0, 5e-15, st, _terms(mesh, mat), "Heun", seed=seed, member=i)
            members.append((it, st))
        return dict(case=case, batch=M.StochasticBatch(members, fused=True), states=[s for _, s in members])
    mat = MATERIALS[case["material"]]
    mesh = M.Mesh(case["nx"], case["ny"], case["nz"], *mat["cell"])
    if kind == "tensor":
        # other inputs for another seed: the cell's height
        mesh.dz *= 1.0 + 0.2 * float(_uniform(seed, 1)[0])
        return dict(case=case, mesh=mesh)
    m = magnetisation(case, seed)
    state = M.State(mesh, mat["Ms"], _host(m), precision=case["precision"])
    out = dict(case=case, state=state)
    if kind == "minimize":
        out["m0"] = np.asfortranarray(_host(m))
        out["solver"] = M.LBFGS_Minimizer(_terms(mesh, mat, case["demag"]), maxiter=case["iterations"])
        return out
    if kind == "field":
        state.set_stream(1)  # the default stream (cudaStreamLegacy), where m comes from and H is used
        out["llg"] = M.LLGIntegrator(mat["alpha"], _terms(mesh, mat))
        out["m"] = m.to(torch.float64 if case["precision"] == "fp64" else torch.float32)
        out["H"] = torch.empty_like(out["m"])
        return out
    h = _step_size(case)
    llg = M.LLGIntegrator(mat["alpha"], _terms(mesh, mat), case["scheme"], hmax=h)
    c = llg.controller_state()
    c[0] = c[3] = h
    llg.set_controller_state(c)
    out["llg"] = llg
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        for _ in range(case["steps"]):
            state["llg"].step(state["state"])
        return _device_m(state["state"])
    if kind == "field":
        state["llg"].heff_device(state["state"], state["m"].data_ptr(), state["H"].data_ptr())
        if case["energy"]:
            return {"H": state["H"], "E": state["llg"].Eeff_in_J(state["state"])}
        return {"H": state["H"]}
    if kind == "tensor":
        return M.DemagField(state["mesh"]).spectral_tensor()
    if kind == "minimize":
        state["state"].m = state["m0"]
        e = state["solver"].minimize(state["state"])
        return {"E": e, "m": _device_m(state["state"])}
    if kind == "ensemble":
        state["batch"].steps(case["steps"])
        return [_device_m(s) for s in state["states"]]
    net, B, H, W = state["net"], case["B"], case["H"], case["W"]
    if kind == "train":
        loss = net.train_step(state["x"].data_ptr(), state["t"].data_ptr(), B, H, W, 1e-4)
        return {"loss": loss, "grad": net.grad}
    return net.forward(state["x"].data_ptr(), B, H, W)


# ------------------------------------------------------------------------------------------------ work
def _evaluation(nx, ny, nz, demag=True):
    """Operations of one field evaluation: the pruned transforms, the tensor product and the local terms."""
    f = 100.0 * nx * ny * nz
    if demag:
        px, py, pz = 2 * nx, 2 * ny, 1 if nz == 1 else 2 * nz
        f += 6 * ny * nz * 2.5 * px * math.log2(px) + 6 * nz * (nx + 1) * 5.0 * py * math.log2(py)
        f += 6 * (nx + 1) * py * 5.0 * pz * math.log2(pz) + 30.0 * (nx + 1) * py * pz
    return f


def _tensor_values(nx, ny, nz):
    return (4 if nz == 1 else 6) * (nx + 1) * (ny + 1) * (1 if nz == 1 else nz + 1)


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        b = f = 0.0
        for nx, ny in _members(case, 0):
            b += 48.0 * nx * ny + 4.0 * _tensor_values(nx, ny, 1)
            f += 2 * case["steps"] * (_evaluation(nx, ny, 1) + 500.0 * nx * ny)
        return {"bytes": b, "flops": f}
    if kind in ("train", "propose"):
        P = case["B"] * case["H"] * case["W"]
        f = 0.0
        for ci, co, lv in _UNET:
            f += 2.0 * 9 * ci * co * P / 4 ** lv
        n = sum(9 * ci * co + co for ci, co, _ in _UNET)
        if kind == "train":
            return {"bytes": P * (8 + 3) * 4.0 + n * 4.0 * 8, "flops": 3 * f}
        return {"bytes": P * (8 + 3) * 4.0 + n * 4.0, "flops": f}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    N = nx * ny * nz
    if kind == "tensor":
        v = _tensor_values(nx, ny, nz)
        return {"bytes": 8.0 * v, "flops": 27.0 * 200 * N * (4 if nz == 1 else 6)}
    r = 8.0 if case["precision"] == "fp64" else 4.0
    T = r * _tensor_values(nx, ny, nz)
    if kind == "field":
        k = 2 if case["energy"] else 1
        return {"bytes": 6.0 * N * r + T, "flops": k * _evaluation(nx, ny, nz)}
    if kind == "minimize":
        return {"bytes": 48.0 * N + (T if case["demag"] else 0.0),
                "flops": case["iterations"] * (_evaluation(nx, ny, nz, case["demag"]) + 100.0 * N)}
    stages = {"RKF45": 6, "DP45": 7, "BS23": 4}[case["scheme"]]
    return {"bytes": 48.0 * N + T, "flops": case["steps"] * stages * (_evaluation(nx, ny, nz) + 100.0 * N)}


# ------------------------------------------------------------------------------------------------ exact
def _ratio(n, d):
    """n / d, and 0 where d = 0 (the terms' limit there)."""
    return torch.where(d != 0, n / torch.where(d != 0, d, torch.ones_like(d)), torch.zeros_like(n))


def _newell_f(x, y, z):
    x2, y2, z2 = x * x, y * y, z * z
    R = (x2 + y2 + z2).sqrt()
    return (y / 2 * (z2 - x2) * torch.asinh(_ratio(y, (x2 + z2).sqrt())) + z / 2 * (y2 - x2) * torch.asinh(_ratio(z, (x2 + y2).sqrt()))
            - x * y * z * torch.atan(_ratio(y * z, x * R)) + (2 * x2 - y2 - z2) * R / 6)


def _newell_g(x, y, z):
    x2, y2, z2 = x * x, y * y, z * z
    R = (x2 + y2 + z2).sqrt()
    return (x * y * z * torch.asinh(_ratio(z, (x2 + y2).sqrt())) + y / 6 * (3 * z2 - y2) * torch.asinh(_ratio(x, (y2 + z2).sqrt()))
            + x / 6 * (3 * z2 - x2) * torch.asinh(_ratio(y, (x2 + z2).sqrt())) - z * z2 / 6 * torch.atan(_ratio(x * y, z * R))
            - z * y2 / 2 * torch.atan(_ratio(x * z, y * R)) - z * x2 / 2 * torch.atan(_ratio(y * z, x * R)) - x * y * R / 3)


def _second_difference(v):
    for a in range(3):
        n = v.shape[a]
        v = 2 * v.narrow(a, 1, n - 2) - v.narrow(a, 0, n - 2) - v.narrow(a, 2, n - 2)
    return v


def _triangle_rule(n):
    """Gauss nodes and weights of the weight 1 - |t| on [-1, 1] (Golub-Welsch on its moments' recurrence)."""
    t, w = np.polynomial.legendre.leggauss(64)
    t, w = np.concatenate([(t - 1) / 2, (t + 1) / 2]), np.concatenate([w, w]) / 2
    w = w * (1 - np.abs(t))
    p0, p1, b = np.zeros_like(t), np.ones_like(t), []
    for _ in range(n):
        s1 = np.sum(w * p1 * p1)
        b.append(s1)
        p0, p1 = p1, t * p1 - (0 if len(b) == 1 else b[-1] / b[-2]) * p0
    J = np.diag([math.sqrt(b[i + 1] / b[i]) for i in range(n - 1)], 1)
    ev, V = np.linalg.eigh(J + J.T)
    return ev, V[0] ** 2 * b[0]


def _octant_tensor(nx, ny, nz, cell):
    """The six components (xx, xy, xz, yy, yz, zz) of the cell-averaged demagnetising tensor, H = N M, at offsets
    0..nx, 0..ny, 0..nz: Newell's closed form near the origin, Gauss quadrature of the dipole field further away
    (where the closed form cancels)."""
    d = [float(c) for c in cell]
    n = (nx + 1, ny + 1, nz + 1)
    axis = [torch.arange(n[a], dtype=torch.float64, device="cuda") for a in range(3)]
    X, Y, Z = (axis[a].reshape([-1 if b == a else 1 for b in range(3)]) * d[a] for a in range(3))
    N = torch.zeros((6,) + n, dtype=torch.float64, device="cuda")
    t, w = _triangle_rule(6)
    vol = d[0] * d[1] * d[2] / (4 * math.pi)
    for i in range(6):
        for j in range(6):
            for k in range(6):
                x, y, z = X + t[i] * d[0], Y + t[j] * d[1], Z + t[k] * d[2]
                r2 = x * x + y * y + z * z
                i3 = (w[i] * w[j] * w[k] * vol) * r2.rsqrt() / r2
                i5 = 3 * i3 / r2
                N[0] += i5 * (x * x) - i3
                N[1] += i5 * (x * y)
                N[2] += i5 * (x * z)
                N[3] += i5 * (y * y) - i3
                N[4] += i5 * (y * z)
                N[5] += i5 * (z * z) - i3
    s = max(d)  # unit of length of the closed form
    near = [min(n[a], int(math.ceil(8 * s / d[a])) + 1) for a in range(3)]
    u = [c / s for c in d]
    c = [torch.arange(-1, near[a] + 1, dtype=torch.float64, device="cuda") * u[a] for a in range(3)]
    gx, gy, gz = torch.meshgrid(c[0], c[1], c[2], indexing="ij")
    k = -1.0 / (4 * math.pi * u[0] * u[1] * u[2])
    sl = (slice(0, near[0]), slice(0, near[1]), slice(0, near[2]))
    N[(0,) + sl] = k * _second_difference(_newell_f(gx, gy, gz))
    N[(1,) + sl] = k * _second_difference(_newell_g(gx, gy, gz))
    N[(2,) + sl] = k * _second_difference(_newell_g(gx, gz, gy))
    N[(3,) + sl] = k * _second_difference(_newell_f(gy, gz, gx))
    N[(4,) + sl] = k * _second_difference(_newell_g(gy, gz, gx))
    N[(5,) + sl] = k * _second_difference(_newell_f(gz, gx, gy))
    return N


_ODD = [(), (0, 1), (0, 2), (), (1, 2), ()]


def _spectrum(nx, ny, nz, cell):
    """Real spectral tensor, six components on [Pz][Py][nx + 1]."""
    N = _octant_tensor(nx, ny, nz if nz > 1 else 0, cell)
    out = []
    for c in range(6):
        g = N[c]
        for a, n in enumerate((nx, ny, nz)):
            if a == 2 and nz == 1:
                if 2 in _ODD[c]:
                    g = torch.zeros_like(g)
                continue
            odd = a in _ODD[c]
            if odd:  # vanishes on the plane through the origin and, on the periodic grid, half a period away
                g = g.clone()
                g.select(a, 0).zero_()
                g.select(a, n).zero_()
            g = torch.cat([g, (-1.0 if odd else 1.0) * g.narrow(a, 1, n - 1).flip(a)], dim=a)
        out.append(torch.fft.rfftn(g.permute(2, 1, 0)).real)
    return out


class _Exact:
    """The effective field of a material on one mesh, in 64-bit torch."""

    def __init__(self, nx, ny, nz, mat, demag=True):
        self.n, self.mat, self.cell = (nx, ny, nz), mat, mat["cell"]
        self.S = _spectrum(nx, ny, nz, self.cell) if demag else None

    def demag(self, M_):
        nx, ny, nz = self.n
        s = (1 if nz == 1 else 2 * nz, 2 * ny, 2 * nx)
        F = [torch.fft.rfftn(M_[c], s=s) for c in range(3)]
        S = self.S
        H = torch.empty_like(M_)
        for a, row in enumerate(((0, 1, 2), (1, 3, 4), (2, 4, 5))):
            H[a] = torch.fft.irfftn(F[0] * S[row[0]] + F[1] * S[row[1]] + F[2] * S[row[2]], s=s)[:nz, :ny, :nx]
        return H

    @staticmethod
    def _shift(m, axis, by):
        """Neighbour along x (axis 0), y, z; zero outside the mesh."""
        dim = m.dim() - 1 - axis
        out, n = torch.zeros_like(m), m.shape[dim]
        if by > 0:
            out.narrow(dim, 0, n - 1).copy_(m.narrow(dim, 1, n - 1))
        else:
            out.narrow(dim, 1, n - 1).copy_(m.narrow(dim, 0, n - 1))
        return out

    def laplace(self, m, edges):
        """Seven-point Laplacian; `edges`: without the missing neighbours' part of the centre weight."""
        L = torch.zeros_like(m)
        one = torch.ones_like(m[:1])
        for a in range(3):
            for by in (1, -1):
                inside = self._shift(one, a, by) if edges else one
                L += (self._shift(m, a, by) - inside * m) / self.cell[a] ** 2
        return L

    def fields(self, m, Ms, edges=False):
        """name -> field; Ms a number or a field [nz][ny][nx] (zero where empty)."""
        mat, out = self.mat, {}
        inv = torch.where(Ms > 0, 1 / torch.where(Ms > 0, Ms, torch.ones_like(Ms)), torch.zeros_like(Ms)) if torch.is_tensor(Ms) else 1 / Ms
        if self.S is not None:
            out["demag"] = self.demag(Ms * m)
        out["exchange"] = (2 * mat["A"] / MU0) * inv * self.laplace(m, edges)
        if "D" in mat:
            d = [(self._shift(m, a, 1) - self._shift(m, a, -1)) / (2 * self.cell[a]) for a in range(3)]
            h = torch.stack([-d[0][2], -d[1][2], (d[0][0] + d[1][1] + d[2][2]) - d[2][2]])
            out["dmi"] = (2 * mat["D"] / MU0) * inv * h
        if "Ku" in mat:
            h = torch.zeros_like(m)
            h[2] = (2 * mat["Ku"] / MU0) * inv * m[2]
            out["uniaxial"] = h
        if "K1" in mat:
            q = m * m
            out["cubic"] = (-2 * mat["K1"] / MU0) * inv * (q.sum(0, keepdim=True) - q) * m
        if "H" in mat:
            out["zeeman"] = torch.tensor(mat["H"], dtype=m.dtype, device=m.device).reshape(3, 1, 1, 1).expand_as(m)
        return out

    def heff(self, m, Ms):
        return sum(self.fields(m, Ms).values())

    def energy(self, m, Ms):
        e = 0.0
        for name, h in self.fields(m, Ms, edges=True).items():
            e += {"cubic": -0.25, "zeeman": -1.0}.get(name, -0.5) * float((Ms * (h * m).sum(0)).sum())
        return MU0 * e * self.cell[0] * self.cell[1] * self.cell[2]

    def rhs(self, m, Ms, h_th=None):
        H = self.heff(m, Ms)
        if h_th is not None:
            H = H + h_th
        a = self.mat["alpha"]
        mxh = torch.linalg.cross(m, H, dim=0)
        return -GAMMA / (1 + a * a) * (mxh + a * torch.linalg.cross(m, mxh, dim=0))


_TABLEAU = {
    "RKF45": ([[], [1 / 4], [3 / 32, 9 / 32], [1932 / 2197, -7200 / 2197, 7296 / 2197], [439 / 216, -8, 3680 / 513, -845 / 4104],
               [-8 / 27, 2, -3544 / 2565, 1859 / 4104, -11 / 40]], [16 / 135, 0, 6656 / 12825, 28561 / 56430, -9 / 50, 2 / 55]),
    "DP45": ([[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9], [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
              [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656]],
             [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]),
    "BS23": ([[], [1 / 2], [0, 3 / 4]], [2 / 9, 1 / 3, 4 / 9]),
}


def _unit(m):
    n = m.square().sum(0, keepdim=True).sqrt()
    return torch.where(n > 0, m / torch.where(n > 0, n, torch.ones_like(n)), torch.zeros_like(m))


def _philox_normals(seed, member, index, cells):
    """Three standard normals per cell from Philox-4x32-10 (Salmon et al., SC'11) and the Box-Muller transform."""
    MASK = 0xFFFFFFFF

    def mul(a, b):  # 32 x 32 -> high, low
        lo, hi = a * (b & 0xFFFF), a * (b >> 16)
        s = lo + ((hi & 0xFFFF) << 16)
        return ((hi >> 16) + (s >> 32)) & MASK, s & MASK

    def block(c, k0, k1):
        for _ in range(10):
            h0, l0 = mul(0xD2511F53, c[0])
            h1, l1 = mul(0xCD9E8D57, c[2])
            c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
            k0, k1 = (k0 + 0x9E3779B9) & MASK, (k1 + 0xBB67AE85) & MASK
        return c

    cell = torch.arange(cells, dtype=torch.int64, device="cuda")
    zero = torch.zeros_like(cell)
    k0, k1 = (seed & MASK) ^ ((member * 0x9E3779B9) & MASK), (seed >> 32) & MASK
    u = []
    for flip in (0, 0x80000000):
        r = block([cell, zero | flip, zero | index, zero], k0, k1)
        u += [(((r[2 * i] << 21) ^ (r[2 * i + 1] >> 11)).double() + 1.0) / 2.0 ** 53 for i in range(2)]
    r1, r2 = (-2 * u[0].log()).sqrt(), (-2 * u[2].log()).sqrt()
    return torch.stack([r1 * (2 * math.pi * u[1]).cos(), r1 * (2 * math.pi * u[1]).sin(), r2 * (2 * math.pi * u[3]).cos()])


_UNET = [(8, 32, 0), (32, 32, 0), (32, 64, 1), (64, 64, 1), (64, 128, 2), (128, 128, 2), (192, 64, 1), (96, 32, 0), (32, 3, 0)]


def _unet_exact(case, seed):
    F = torch.nn.functional
    net = UNet(8, seed=seed)  # its initial parameters are the input; nothing of it computes here
    layers = net.layers
    p = torch.from_numpy(_unet_params(net, seed)).double().cuda().requires_grad_(True)
    x, t = _unet_inputs(case, seed)
    x, t = x.double(), t.double()

    def conv(i, v):
        L = layers[i]
        w = p[L.woff:L.boff].reshape(L.cout, 3, 3, L.cin).permute(0, 3, 1, 2)
        v = F.conv2d(v, w, p[L.boff:L.boff + L.cout], padding=1)
        return v.relu() if L.relu else v

    up = lambda v: F.interpolate(v, scale_factor=2, mode="nearest")  # noqa: E731
    e1 = conv(1, conv(0, x))
    e2 = conv(3, conv(2, F.avg_pool2d(e1, 2)))
    b = conv(5, conv(4, F.avg_pool2d(e2, 2)))
    u1 = conv(7, torch.cat([up(conv(6, torch.cat([up(b), e2], 1))), e1], 1))
    y = x[:, :3] + conv(8, u1)
    y = (y / y.square().sum(1, keepdim=True).sqrt()).permute(0, 2, 3, 1).reshape(-1, 3)
    if case["kind"] == "propose":
        return y.detach()
    loss = (y - t).square().sum(1).mean()
    loss.backward()
    return {"loss": float(loss), "grad": p.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "propose"):
        return _unet_exact(case, seed)
    if kind == "minimize":
        return None  # the line search's decisions belong to the method: there is no value without restating it whole
    if kind == "ensemble":
        mat = MATERIALS["cobalt_film"]
        out = []
        dt, dV = 5e-15, mat["cell"][0] * mat["cell"][1] * mat["cell"][2]
        sigma = math.sqrt(2 * (mat["alpha"] * KB * 300.0) / (GAMMA * MU0 * mat["Ms"] * dV) / dt)
        known = {}
        for i, (nx, ny) in enumerate(_members(case, seed)):
            m = magnetisation(dict(nx=nx, ny=ny, nz=1, start="smooth"), seed + 1000 * i)
            ex = known.setdefault((nx, ny), None) or _Exact(nx, ny, 1, mat)
            known[(nx, ny)] = ex
            noise = lambda q: sigma * _philox_normals(seed, i, q, nx * ny).reshape(3, 1, ny, nx)  # noqa: E731
            for q in range(case["steps"]):
                k1 = dt * ex.rhs(m, mat["Ms"], noise(q))
                k2 = dt * ex.rhs(m + k1, mat["Ms"], noise(q + 1))
                m = _unit(m + (k1 + k2) / 2)
            out.append(m)
        return out
    mat = dict(MATERIALS[case["material"]])
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if kind == "tensor":
        dx, dy, dz = mat["cell"]
        dz *= 1.0 + 0.2 * float(_uniform(seed, 1)[0])
        S = _spectrum(nx, ny, nz, (dx, dy, dz))
        keep = (0, 1, 3, 5) if nz == 1 else range(6)
        return torch.stack([S[c][:nz + 1 if nz > 1 else 1, :ny + 1] for c in keep]).cpu().numpy()
    ex = _Exact(nx, ny, nz, mat)
    m = _unit(magnetisation(case, seed))
    Ms = mat["Ms"]
    if kind == "field":
        out = {"H": ex.heff(m, Ms)}
        if case["energy"]:
            out["E"] = ex.energy(m, Ms)
        return out
    if case["geometry"] == "disc":
        Ms = Ms * (m.square().sum(0) > 0).to(torch.float64)
    a, b = _TABLEAU[case["scheme"]]
    h = _step_size(case)
    for _ in range(case["steps"]):
        k = []
        for row in a:
            ms = m
            for c, kj in zip(row, k):
                ms = ms + c * kj
            k.append(h * ex.rhs(ms, Ms))
        for c, kj in zip(b, k):
            m = m + c * kj
        m = _unit(m)
    return m
