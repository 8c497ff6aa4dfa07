"""Performance cases of the solver: what its users run, through its public entry points.

Every case is a dict of plain values.  ``prepare`` builds what a program has in hand before the call (a
state on the GPU, the solver context or the network), ``run`` is one pass through the entry point,
``work`` counts the bytes and operations the pass cannot do without and ``exact`` is its result in 64 bits
from plain torch, with every line operator as a dense matrix.

Flows (sizes from the repository's configurations, studies and tests):

* ``vortex``   2-D isentropic vortex, o8 differences and o10 filter, z collapsed: the smallest calls
* ``box``      periodic Taylor-Green box, o8 differences and o10 filter: the headline configuration
* ``layer``    temporal mixing layer: o8 in x and z, compact o6 in y, type-201 rows and a sponge in y
* ``pulse``    pressure pulse in an open box: o4 one-sided closures and type-201 rows on all six faces
* ``compact``  periodic box on the reference's compact o6 derivatives and filters in all directions
* ``closure``  periodic coarse box with the learned closure in the flux pass
"""
import math

import numpy as np
import torch

from public_b200.autograd import objective
from public_b200.closure import ClosureMLP
from public_b200.cruna import Cruna, Settings

DEV = "cuda:0"
GAMMA, PR, S1 = 1.4, 0.71, 110.4
HID, NIN, NOUT = 64, 12, 6


def listed():
    return [
        # a 2-D run of the vortex configuration: short launches, step graphs, an empty z direction
        dict(name="vortex_run_256", kind="vortex", loop="direct", n1=256, n2=256, n3=1, steps=16),
        # one direct and one adjoint loop step of the benchmark's grid (RK4 and the filters)
        dict(name="box_direct_256", kind="box", loop="direct", n1=256, n2=256, n3=256, steps=1),
        dict(name="box_adjoint_256", kind="box", loop="adjoint", n1=256, n2=256, n3=256, steps=1),
        # the FP32-stencil precision on the same grid, a direct and an adjoint step
        dict(name="box_fp32_pair_256", kind="box", loop="pair", n1=256, n2=256, n3=256, steps=1, precision="fp32"),
        # the mixing layer's loops on the grid of its profiles
        dict(name="layer_direct_256", kind="layer", loop="direct", n1=256, n2=192, n3=128, steps=1),
        dict(name="layer_adjoint_256", kind="layer", loop="adjoint", n1=256, n2=192, n3=128, steps=1),
        # the gradient of its plane objective through the autograd wrapper: discrete adjoint, checkpointing
        dict(name="layer_gradient_128", kind="layer", loop="gradient", n1=128, n2=96, n3=64, steps=4),
        # the reference's unit-test pulse on its odd grid
        dict(name="pulse_run_60", kind="pulse", loop="direct", n1=60, n2=65, n3=70, steps=8),
        # the reference's own compact schemes in every direction
        dict(name="compact_direct_128", kind="compact", loop="direct", n1=128, n2=120, n3=96, steps=2),
        # the closure-augmented coarse run
        dict(name="closure_run_64", kind="closure", loop="direct", n1=64, n2=64, n3=64, steps=4),
        # inference on the training set of the closure study, and a stretch of its training
        dict(name="mlp_forward_2m", kind="mlp", loop="forward", samples=2_000_000),
        dict(name="mlp_train_4096", kind="mlp", loop="train", samples=65_536, batch=4096, steps=32),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind, loop = rng.choice([("vortex", "direct"), ("box", "direct"), ("box", "adjoint"), ("box", "pair"),
                             ("layer", "direct"), ("layer", "adjoint"), ("layer", "gradient"), ("pulse", "direct"),
                             ("compact", "direct"), ("closure", "direct"), ("mlp", "forward"), ("mlp", "train")])
    if kind == "mlp":
        if loop == "forward":
            return dict(kind=kind, loop=loop, samples=size(1, 2_000_000))
        return dict(kind=kind, loop=loop, samples=size(4096, 262_144), batch=128 * rng.randint(1, 32),
                    steps=rng.randint(4, 32))
    lo, hi = {"vortex": ((32, 32, 1), (256, 256, 1)), "box": ((24, 24, 24), (256, 256, 256)),
              "layer": ((24, 32, 16), (256, 192, 128)), "pulse": ((20, 20, 20), (96, 96, 96)),
              "compact": ((20, 20, 20), (128, 128, 128)), "closure": ((16, 16, 16), (96, 96, 96))}[kind]
    if loop == "gradient":
        hi = (128, 96, 64)
    n1, n2, n3 = (size(a, b) for a, b in zip(lo, hi))
    case = dict(kind=kind, loop=loop, n1=n1, n2=n2, n3=n3, steps=1 if kind == "box" or loop == "adjoint" else rng.randint(1, 4))
    if loop == "pair":
        case["precision"] = "fp32"
    if kind == "vortex":
        case["steps"] = rng.randint(2, 16)
    return case


# ---- inputs --------------------------------------------------------------------------------------
class _Rand:
    """Seeded inputs: smooth fields of a few Fourier modes, and white noise."""

    def __init__(self, seed):
        self.small = np.random.Generator(np.random.PCG64(seed))
        self.gen = torch.Generator(device=DEV).manual_seed(int(seed) + 1)

    def noise(self, *shape, dtype=torch.float64):
        return torch.randn(*shape, generator=self.gen, device=DEV, dtype=dtype)

    def smooth(self, n, modes=4, kmax=3):
        f = torch.zeros(n[2], n[1], n[0], device=DEV, dtype=torch.float64)
        for _ in range(modes):
            w = []
            for m in n:
                k, ph = int(self.small.integers(0, kmax + 1)), float(self.small.uniform(0, 2 * math.pi))
                w.append(torch.cos(k * 2 * math.pi / m * torch.arange(m, device=DEV, dtype=torch.float64) + ph))
            f += float(self.small.uniform(0.5, 1.0)) / modes * w[2][:, None, None] * w[1][None, :, None] * w[0][None, None, :]
        return f


def _axis(n, lo, step, dim):
    shape = [1, 1, 1]
    shape[dim] = n
    return (lo + step * torch.arange(n, device=DEV, dtype=torch.float64)).view(shape)


def _box_rows(n, faces):
    """Boundary-table rows of type 201 on the given faces (direction, end, outward sign)."""
    rows = []
    for d, end in faces:
        box, k = [1, n[0], 1, n[1], 1, n[2]], [0.0, 0.0, 0.0]
        box[2 * d] = box[2 * d + 1] = 1 if end == 0 else n[d]
        k[d] = -1.0 if end == 0 else 1.0
        rows.append([201, *box, *k])
    return rows


def _flow(case, rand):
    """Initial state (rho, rho u, rho v, rho w, p) as (5, n3, n2, n1), and the solver's settings."""
    kind = case["kind"]
    n = (case["n1"], case["n2"], case["n3"])
    X = Y = Z = None
    s = dict(n=n, gamma=GAMMA, R=1.0, W=1.0, Pr=PR, di_freq=(1, 1, 1), ai_freq=(1, 1, 1), alpha=0.0, strength=0.2)
    one = torch.ones(n[2], n[1], n[0], device=DEV, dtype=torch.float64)
    if kind == "vortex":
        dx = (10.0 / n[0], 10.0 / n[1], 1.0)
        X, Y = _axis(n[0], -5.0, dx[0], 2), _axis(n[1], -5.0, dx[1], 1)
        c0 = math.sqrt(GAMMA)
        f = torch.exp(0.5 * (1.0 - X ** 2 - Y ** 2)) * one
        amp = 5.0 / (2 * math.pi)
        T = 1.0 - (GAMMA - 1.0) * 25.0 / (8 * GAMMA * math.pi ** 2) * f ** 2
        rho = T ** (1 / (GAMMA - 1)) * (1 + 0.01 * rand.smooth(n))
        p = rho * T
        vel = [0.5 * c0 - amp * Y * f, amp * X * f, 0.05 * rand.smooth(n)]
        s.update(x0=(-5.0, -5.0, 0.0), x1=(5.0, 5.0, 1.0), diff=("o8_e_c_p", "o8_e_c_p", "empty"),
                 filt=("o10_e_c_p", "o10_e_c_p", "empty"), mu0=0.5 * c0 / 1000.0, T0=1.0)
    elif kind in ("box", "compact", "closure"):
        mach = 0.3 if kind == "closure" else 0.1
        L = 2 * math.pi
        dx = tuple(L / m for m in n)
        X, Y, Z = _axis(n[0], 0.0, dx[0], 2), _axis(n[1], 0.0, dx[1], 1), _axis(n[2], 0.0, dx[2], 0)
        p0 = 1.0 / (GAMMA * mach ** 2)
        rho = 1 + 1e-4 * rand.noise(n[2], n[1], n[0]) + 0.01 * rand.smooth(n)
        vel = [torch.sin(X) * torch.cos(Y) * torch.cos(Z) + 0.1 * rand.smooth(n, kmax=4),
               -torch.cos(X) * torch.sin(Y) * torch.cos(Z) + 0.1 * rand.smooth(n, kmax=4), 0.1 * rand.smooth(n, kmax=4)]
        p = p0 + (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0) / 16.0 * one
        s.update(x1=(L, L, L), diff=("o8_e_c_p",) * 3, filt=("o10_e_c_p",) * 3, mu0=1.0 / 1600.0, T0=p0,
                 precision=case.get("precision", "fp64"))
        if kind == "compact":
            s.update(diff=("o6_i_c_p",) * 3, filt=("o6_i_c_p",) * 3, alpha=0.35)
    elif kind == "layer":
        Ls = (80.0, 60.0, 40.0)
        dx = (Ls[0] / n[0], Ls[1] / (n[1] - 1), Ls[2] / n[2])
        Y = _axis(n[1], -30.0, dx[1], 1)
        dU = 0.8 * math.sqrt(GAMMA)
        vel = [0.5 * dU * torch.tanh(Y) + 0.05 * dU * rand.smooth(n) + 1e-3 * dU * rand.noise(n[2], n[1], n[0])]
        vel += [0.05 * dU * rand.smooth(n) + 1e-3 * dU * rand.noise(n[2], n[1], n[0]) for _ in range(2)]
        rho = 1 + 0.02 * rand.smooth(n)
        p = 1 + 0.02 * rand.smooth(n)
        rows = _box_rows(n, [(1, 0), (1, 1)]) + [[400, 1, n[0], 1, n[1], 1, n[2], 0, 0, 0]]
        s.update(x0=(0.0, -30.0, 0.0), x1=(80.0, 30.0, 40.0), diff=("o8_e_c_p", "o6_i_c_o", "o8_e_c_p"),
                 filt=("o10_e_c_p", "o10_i_c_o", "o10_e_c_p"), mu0=dU / 500.0, T0=1.0, bc=np.array(rows),
                 sponge_length=(0.0, min(20, n[1] // 4) * dx[1], 0.0), sponge_amplitude=1.0)
    else:  # pulse
        L = 6.283185307
        dx = tuple(L / (m - 1) for m in n)
        X, Y, Z = _axis(n[0], 0.0, dx[0], 2), _axis(n[1], 0.0, dx[1], 1), _axis(n[2], 0.0, dx[2], 0)
        r2 = (X - 3.14) ** 2 + (Y - 3.14) ** 2 + (Z - 3.14) ** 2
        p = 101325.0 + 1000.0 * torch.exp(-r2 / (2 * (10 / 2.3548 * dx[0]) ** 2)) + 100.0 * rand.smooth(n)
        rho = 1.193847801511275 * (p / 101325.0) ** (1 / GAMMA)
        vel = [rand.smooth(n) for _ in range(3)]
        s.update(x1=(L, L, L), diff=("o4_e_c_o",) * 3, filt=("empty",) * 3, R=8.3144598, W=0.0289647, mu0=0.0,
                 T0=273.0, bc=np.array(_box_rows(n, [(d, e) for d in range(3) for e in (0, 1)])))
    q = torch.stack([rho * one] + [rho * v * one for v in vel] + [p * one])
    speed = (q[1:4].square().sum(0).sqrt() / q[0] + (GAMMA * q[4] / q[0]).sqrt()).max().item()
    s["dt"] = 0.5 * min(d for d, m in zip(dx, n) if m > 1) / speed
    return q, s, dx


def _params(rand):
    """Network parameters W1, b1, W2, b2, W3, b3 (uniform +-1/sqrt(fan in)) in the order of ClosureMLP."""
    sizes = [(HID * NIN, NIN), (HID, NIN), (HID * HID, HID), (HID, HID), (NOUT * HID, HID), (NOUT, HID)]
    return np.concatenate([rand.small.uniform(-1, 1, m) / math.sqrt(f) for m, f in sizes]).astype(np.float32)


def _scaling(T0, delta):
    return ([0.0] * 9 + [1.0, T0, delta], [1.0] * 9 + [0.05, 0.05 * T0, 1.0], [1e-3] * NOUT)


def _samples(rand, n):
    """Closure features (velocity gradients, rho, T, filter width) and stresses of a plausible size."""
    X = torch.empty(n, NIN, device=DEV, dtype=torch.float32)
    X[:, :9] = rand.noise(n, 9, dtype=torch.float32)
    X[:, 9] = 1 + 0.05 * rand.noise(n, dtype=torch.float32)
    X[:, 10] = 8 * (1 + 0.05 * rand.noise(n, dtype=torch.float32))
    X[:, 11] = 0.1
    g = X[:, :9].reshape(n, 3, 3)
    t = 1e-3 * torch.matmul(g, g.transpose(1, 2)) * X[:, 9].view(n, 1, 1)
    Y = torch.stack([t[:, i, j] for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))], 1).contiguous()
    return X, Y + 1e-4 * rand.noise(n, NOUT, dtype=torch.float32)


class State:
    """What a program holds between calls: the case, its tensors, and the solver or network it made."""

    def __init__(self, case):
        self.case = case


def _inputs(case, seed):
    st = State(case)
    rand = _Rand(seed)
    if case["kind"] == "mlp":
        st.params = _params(rand)
        st.scaling = _scaling(8.0, 0.1)
        st.X, st.Y = _samples(rand, case["samples"])
        return st
    st.q0, st.settings, st.dx = _flow(case, rand)
    st.qref = st.q0.clone() if st.settings.get("bc") is not None else None
    n = st.settings["n"]
    if case["loop"] in ("adjoint", "pair"):
        st.qs0 = torch.stack([1e-3 * rand.smooth(n, modes=6, kmax=4) for _ in range(5)])
    if case["loop"] == "gradient":
        st.f0 = torch.stack([1e-3 * rand.smooth(n) for _ in range(5)])
        st.index = int(round(25.0 / st.dx[1])) + 1
    if case["kind"] == "closure":
        st.params = _params(rand)
        st.delta = st.dx[0]
        st.scaling = _scaling(st.settings["T0"], st.delta)
    return st


def prepare(case, seed):
    st = _inputs(case, seed)
    if case["kind"] == "mlp" or case["kind"] == "closure":
        st.mlp = ClosureMLP(0, seed=0)
        st.mlp.params = st.params
        st.mlp.set_scaling(*st.scaling)
        if case["kind"] == "mlp":
            return st
    qref = None if st.qref is None else np.asfortranarray(st.qref.cpu().numpy().transpose(3, 2, 1, 0))
    st.solver = Cruna(Settings.from_dict(st.settings), qref=qref)
    st.stream = torch.cuda.ExternalStream(st.solver.stream_handle(), device=DEV)
    if case["kind"] == "closure":
        st.solver.set_closure(st.mlp, st.delta)
    if case["loop"] == "gradient":
        st.solver.set_adjoint_mode(1)
        st.goal = Cruna.objective("plane_p2", normal=2, index=st.index, p_inf=1.0)
    st.q = torch.empty_like(st.q0)
    st.qs = torch.empty_like(st.q0)
    torch.cuda.synchronize()
    return st


# ---- one pass ------------------------------------------------------------------------------------
def run(st):
    case = st.case
    loop = case["loop"]
    if loop == "forward":
        return st.mlp.forward(st.X)
    if loop == "train":
        st.mlp.params = st.params  # a fresh start: sets the parameters and clears Adam's moments
        loss = st.mlp.train(st.X, st.Y, batch=case["batch"], steps=case["steps"], lr=1e-3, seed=7)
        return {"loss": loss, "params": st.mlp.params}
    if loop == "gradient":
        q0, f = st.q0.view(-1).clone().requires_grad_(), st.f0.view(-1).clone().requires_grad_()
        J = objective(q0, f, st.solver, case["steps"], 2, st.goal)
        J.backward()
        return {"J": J.detach(), "dJ/dq0": q0.grad, "dJ/df": f.grad}
    # the solver works on its own stream: ordered after and before the caller's work, no host wait
    here = torch.cuda.current_stream()
    st.stream.wait_stream(here)
    out = {}
    with torch.cuda.stream(st.stream):
        if loop in ("direct", "pair"):
            st.q.copy_(st.q0)
            st.solver.run_direct_dev(st.q.data_ptr(), 0, case["steps"])
            out["q"] = list(st.q)
        if loop in ("adjoint", "pair"):
            st.qs.copy_(st.qs0)
            st.solver.run_adjoint_dev(st.qs.data_ptr(), st.q0.data_ptr(), None, 1, 1)
            out["qs"] = list(st.qs)
    here.wait_stream(st.stream)
    return out


def work(case):
    """Bytes and operations of a pass.  An RK4 loop step moves at least the states of its stages: each
    stage reads its input (and q0 and the accumulated slope from the second on) and writes the next input
    and the slope, the filters read and write the state: 760 bytes a point; the adjoint reads the direct
    state in each stage as well: 920.  Operations: first derivatives of 42 (adjoint: 21) products."""
    if case["kind"] == "mlp":
        n = case["samples"] if case["loop"] == "forward" else case["batch"] * case["steps"]
        return {"bytes": 4.0 * (NIN + NOUT) * n,
                "flops": 2.0 * (NIN * HID + HID * HID + HID * NOUT) * n * (1 if case["loop"] == "forward" else 3)}
    pts = case["n1"] * case["n2"] * case["n3"]
    direct, adjoint = {"bytes": 760.0, "flops": 4 * 720.0 + 300}, {"bytes": 920.0, "flops": 4 * 420.0 + 300}
    parts = {"direct": [direct], "adjoint": [adjoint], "pair": [direct, adjoint], "gradient": [direct, adjoint]}
    w = {k: pts * case["steps"] * sum(p[k] for p in parts[case["loop"]]) for k in ("bytes", "flops")}
    if case["kind"] == "closure":
        w["flops"] += 4.0 * case["steps"] * pts * 2 * (NIN * HID + HID * HID + HID * NOUT)
    return w


# ---- the same passes in plain torch, 64 bits ------------------------------------------------------
def _banded(n, c, periodic, anti):
    """Matrix of an interior stencil c[m] at offsets +-m (wrapped, or rows that stay inside)."""
    A = torch.zeros(n, n, dtype=torch.float64)
    i = torch.arange(n)
    for m, w in c.items():
        for off, sign in ((m, 1.0), (-m, -1.0 if anti else 1.0)) if m else ((0, 1.0),):
            j = i + off
            ok = torch.ones(n, dtype=torch.bool) if periodic else (j >= 0) & (j < n)
            A[i[ok], j[ok] % n] += sign * w
    return A


def _end_rows(A, rows, sign):
    """Puts one-sided rows at the start and mirrored ones at the end."""
    n = A.shape[0]
    for r, w in enumerate(rows):
        w = torch.tensor(w, dtype=torch.float64)
        A[r] = 0.0
        A[r, :len(w)] = w
        A[n - 1 - r] = 0.0
        A[n - 1 - r, n - len(w):] = sign * w.flip(0)
    return A


def _derivative(scheme, n):
    """First-derivative matrix of a scheme on n points of spacing 1."""
    if scheme == "empty":
        return torch.zeros(n, n, dtype=torch.float64, device=DEV)
    if scheme == "o8_e_c_p":
        return _banded(n, {1: 4 / 5, 2: -1 / 5, 3: 4 / 105, 4: -1 / 280}, True, True).to(DEV)
    if scheme == "o4_e_c_o":
        A = _banded(n, {1: 8.0, 2: -1.0}, False, True)
        return (_end_rows(A, [[-25.0, 48.0, -36.0, 16.0, -3.0], [-3.0, -10.0, 18.0, -6.0, 1.0]], -1.0) / 12).to(DEV)
    third = _banded(n, {0: 1.0, 1: 1 / 3}, scheme == "o6_i_c_p", False)
    A = _banded(n, {1: 7 / 9, 2: 1 / 36}, scheme == "o6_i_c_p", True)
    if scheme == "o6_i_c_o":
        _end_rows(A, [[-17 / 6, 1.5, 1.5, -1 / 6], [-0.75, 0.0, 0.75]], -1.0)
        _end_rows(third, [[1.0, 3.0], [0.25, 1.0, 0.25]], 1.0)
    return torch.linalg.solve(third, A).to(DEV)


def _filter(scheme, n, alpha, strength):
    if scheme == "empty":
        return None
    eye = torch.eye(n, dtype=torch.float64)
    if scheme == "o6_i_c_p":
        c = {0: 11 / 16 + 5 * alpha / 8, 1: (15 / 32 + 17 * alpha / 16) / 2, 2: (-3 / 16 + 3 * alpha / 8) / 2,
             3: (1 / 32 - alpha / 16) / 2}
        return torch.linalg.solve(_banded(n, {0: 1.0, 1: alpha}, True, False), _banded(n, c, True, False)).to(DEV)
    # tenth order at alpha = 0: the identity less the tenth difference / 1024 of the nearest 11 points
    w = [math.comb(10, m) / 1024 for m in range(11)]
    if scheme == "o10_e_c_p":
        F = _banded(n, {0: 1 - w[5], **{m: -(-1) ** m * w[5 + m] for m in range(1, 6)}}, True, False)
        return (eye - strength * (eye - F)).to(DEV)
    F = _banded(n, {0: 1 - w[5], **{m: -(-1) ** m * w[5 + m] for m in range(1, 6)}}, False, False)
    rows = [[1.0]] + [[(j == r) - (-1) ** (j + r) * w[j] for j in range(11)] for r in range(1, 5)]
    return _end_rows(F, rows, 1.0).to(DEV)


def _along(M, f, d):
    """M applied along direction d of a (..., n3, n2, n1) field."""
    if d == 0:
        return f @ M.T
    if d == 1:
        return M @ f
    return (M @ f.reshape(*f.shape[:-3], f.shape[-3], -1)).reshape(f.shape)


class _Plain:
    """The direct and adjoint loop steps in plain torch."""

    def __init__(self, st):
        s = st.settings
        self.s, self.n, self.dx, self.qref = s, s["n"], st.dx, st.qref
        self.unit = [_derivative(s["diff"][d], self.n[d]) for d in range(3)]
        self.D = [M / h for M, h in zip(self.unit, self.dx)]
        self.F = [_filter(s["filt"][d], self.n[d], s["alpha"], s["strength"]) for d in range(3)]
        self.rows = [] if s.get("bc") is None else [[int(v) for v in r] for r in s["bc"]]
        self.net = None
        if hasattr(st, "params"):
            self.net, self.scaling, self.delta = _net(st.params), st.scaling, st.delta

    def d(self, k, f):
        return _along(self.D[k], f, k)

    def faces(self):
        for r in self.rows:
            if r[0] == 201:
                yield (Ellipsis, slice(r[5] - 1, r[6]), slice(r[3] - 1, r[4]), slice(r[1] - 1, r[2])), [-float(v) for v in r[7:10]]

    def shape(self):
        """Strength of the type-400 sponge over y."""
        L, y0, y1 = self.s["sponge_length"][1], self.s["x0"][1], self.s["x1"][1]
        y = _axis(self.n[1], y0, self.dx[1], 1)
        lo = torch.where(y > y0 + L, torch.ones_like(y), 1 - ((y - (y0 + L)) / L) ** 2)
        hi = torch.where(y < y1 - L, torch.ones_like(y), 1 - ((y - (y1 - L)) / L) ** 2)
        return self.s["sponge_amplitude"] * (1 - lo * hi)

    def bc_q(self, q):
        for at, (kx, ky, kz) in self.faces():
            b, a = q[at], self.qref[at]
            r, p = b[0], b[4]
            u = b[1:4] / r
            c = torch.sqrt(GAMMA * p / r)
            d = [a[0] - r, a[1] / a[0] - u[0], a[2] / a[0] - u[1], a[3] / a[0] - u[2], a[4] - p]
            zero = torch.zeros_like(r)
            ls = kx * u[0] + ky * u[1] + kz * u[2]
            R = [kx * d[0] + kz * d[2] - ky * d[3] - kx * d[4] / c ** 2, ky * d[0] - kz * d[1] + kx * d[3] - ky * d[4] / c ** 2,
                 kz * d[0] + ky * d[1] - kx * d[2] - kz * d[4] / c ** 2]
            R = [torch.where(ls < 0, zero, v) for v in R]
            kd = kx * d[1] + ky * d[2] + kz * d[3]
            R4 = torch.where(ls + c < 0, zero, kd + d[4] / (r * c))
            R5 = torch.where(ls - c < 0, zero, -kd + d[4] / (r * c))
            e1 = kx * R[0] + ky * R[1] + kz * R[2] + r / (2 * c) * (R4 + R5)
            e2 = -kz * R[1] + ky * R[2] + 0.5 * kx * (R4 - R5)
            e3 = kz * R[0] - kx * R[2] + 0.5 * ky * (R4 - R5)
            e4 = -ky * R[0] + kx * R[1] + 0.5 * kz * (R4 - R5)
            rn = r + e1
            q = q.clone()
            q[at] = torch.stack([rn, rn * (u[0] + e2), rn * (u[1] + e3), rn * (u[2] + e4), p + 0.5 * r * c * (R4 + R5)])
        return q

    def bc_qs(self, qs, q):
        for at, (kx, ky, kz) in self.faces():
            b, a = qs[at], q[at]
            ds = [-v for v in b]
            c = torch.sqrt(GAMMA * a[4] / a[0])
            gc = (GAMMA - 1) / c
            u = a[1:4] / a[0]
            ku = kx * u[0] + ky * u[1] + kz * u[2]
            kus = kx * ds[1] + ky * ds[2] + kz * ds[3]
            ruus = (ds[0] + u[0] * ds[1] + u[1] * ds[2] + u[2] * ds[3]) / c
            rups = ruus + ds[4] / gc
            zero = torch.zeros_like(c)
            on = ku < 0
            out = [torch.where(on, v, zero) for v in (ds[0] + ku * kus, ds[1] - kx * kus, ds[2] - ky * kus, ds[3] - kz * kus,
                                                      -gc * ruus)]
            for sign in (1.0, -1.0):
                t = torch.where(ku + sign * c < 0, 0.5 * (kus + sign * rups), zero)
                out = [out[0] - ku * t, out[1] + kx * t, out[2] + ky * t, out[3] + kz * t, out[4] + sign * gc * t]
            qs = qs.clone()
            qs[at] = torch.stack([x + y for x, y in zip(b, out)])
        return qs

    def rhs(self, q, force=None):
        s = self.s
        q = self.bc_q(q)
        rho, m, p = q[0], q[1:4], q[4]
        u = m / rho
        WoR = s["W"] / s["R"]
        T = WoR * p / rho
        mu = s["mu0"] * (T / s["T0"]) ** 1.5 * ((s["T0"] + S1) / (T + S1))
        g = [[self.d(k, u[v]) for k in range(3)] for v in range(3)]
        div = g[0][0] + g[1][1] + g[2][2]
        tau = [[mu * (g[v][k] + g[k][v]) - (2 / 3 * mu * div if v == k else 0.0) for k in range(3)] for v in range(3)]
        flux = tau
        if self.net is not None:
            x = [g[v][k] for v in range(3) for k in range(3)] + [rho, T, torch.full_like(T, self.delta)]
            y = _network(self.net, torch.stack([f.reshape(-1) for f in x], 1), self.scaling)
            t = [y[:, i].reshape(T.shape) for i in range(6)]
            at = [[0, 3, 4], [3, 1, 5], [4, 5, 2]]
            flux = [[tau[v][k] - t[at[v][k]] for k in range(3)] for v in range(3)]
        px = [self.d(k, p) for k in range(3)]
        out = [-sum(self.d(k, m[k]) for k in range(3))]
        for v in range(3):
            out.append(-sum(self.d(k, m[k] * u[v]) for k in range(3)) - px[v] + sum(self.d(k, flux[v][k]) for k in range(3)))
        lam = mu * (GAMMA / WoR / (GAMMA - 1) / s["Pr"])
        e = -GAMMA / (GAMMA - 1) * sum(self.d(k, p * u[k]) for k in range(3)) + sum(u[k] * px[k] for k in range(3))
        # the reference differences the heat flux on a spacing of 1
        e = e + sum(_along(self.unit[k], lam * _along(self.unit[k], T, k), k) for k in range(3))
        e = e + sum(tau[v][k] * g[v][k] for v in range(3) for k in range(3))
        out = torch.stack(out + [(GAMMA - 1) * e])
        if force is not None:
            out = out + force
        if any(r[0] == 400 for r in self.rows):
            out = out - self.shape() * (q - self.qref)
        return out

    def rhs_adjoint(self, qs, q):
        qs = self.bc_qs(qs, q)
        u, ir, gm1 = q[1:4] / q[0], 1 / q[0], GAMMA - 1
        gpr = GAMMA * q[4] / (q[0] * gm1)
        r = [torch.zeros_like(ir) for _ in range(5)]
        for k in range(3):
            a, b, c, d, e = (self.d(k, f) for f in qs)
            grad, pk = [b, c, d], self.d(k, q[4])
            r[0] = r[0] + u[k] * (u[0] * b + u[1] * c + u[2] * d) + gpr * u[k] * e + qs[4] * u[k] * ir * pk
            for v in range(3):
                r[1 + v] = r[1 + v] - u[k] * grad[v]
            r[1 + k] = r[1 + k] - a - (u[0] * b + u[1] * c + u[2] * d) - gpr * e - qs[4] * ir * pk
            r[4] = r[4] - gm1 * grad[k] - GAMMA * u[k] * e + gm1 * self.d(k, u[k] * qs[4])
        return torch.stack(r)

    @staticmethod
    def rk4(f, y, dt):
        k1 = f(y)
        k2 = f(y + 0.5 * dt * k1)
        k3 = f(y + 0.5 * dt * k2)
        k4 = f(y + dt * k3)
        return y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)

    def filters(self, q):
        for k in range(3):
            if self.F[k] is not None:
                q = _along(self.F[k], q, k)
        return q

    def direct(self, q, force=None):
        return self.filters(self.bc_q(self.rk4(lambda y: self.rhs(y, force), q, self.s["dt"])))

    def adjoint(self, qs, q):
        return self.filters(self.bc_qs(self.rk4(lambda y: self.rhs_adjoint(y, q), qs, -self.s["dt"]), q))


def _net(params):
    p = torch.from_numpy(params).to(DEV).double()
    cut = np.cumsum([0, HID * NIN, HID, HID * HID, HID, NOUT * HID, NOUT])
    w = [p[a:b] for a, b in zip(cut[:-1], cut[1:])]
    return w[0].view(HID, NIN), w[1], w[2].view(HID, HID), w[3], w[4].view(NOUT, HID), w[5]


def _network(net, x, scaling):
    mean, scale, out = (torch.tensor(np.float32(v), device=DEV).double() for v in scaling)
    W1, b1, W2, b2, W3, b3 = net
    gelu = torch.nn.functional.gelu
    h = gelu(((x - mean) / scale) @ W1.T + b1)
    h = gelu(h @ W2.T + b2)
    return (h @ W3.T + b3) * out


def exact(case, seed):
    if case["loop"] == "train":
        return None  # the order of the mini-batches is the C++ library's shuffle
    st = _inputs(case, seed)
    if case["loop"] == "forward":
        return torch.cat([_network(_net(st.params), x.double(), st.scaling) for x in st.X.split(1 << 18)])
    plain = _Plain(st)
    if case["loop"] == "gradient":
        q0, f = st.q0.clone().requires_grad_(), st.f0.clone().requires_grad_()
        J, q = 0.0, q0
        for _ in range(case["steps"]):
            q = plain.direct(q, f)
            J = J + st.settings["dt"] * st.dx[0] * st.dx[2] * (q[4][:, st.index - 1] - 1.0).square().sum()
        J.backward()
        return {"J": J.detach(), "dJ/dq0": q0.grad.view(-1), "dJ/df": f.grad.view(-1)}
    out = {}
    with torch.no_grad():
        if case["loop"] in ("direct", "pair"):
            q = st.q0
            for _ in range(case["steps"]):
                q = plain.direct(q)
            out["q"] = list(q)
        if case["loop"] in ("adjoint", "pair"):
            out["qs"] = list(plain.adjoint(st.qs0, st.q0))
    return out
