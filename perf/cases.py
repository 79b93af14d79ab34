"""The work that users of this framework have it do, as measurable cases.

Every case goes through the public entry points of `wlc` (the Python mirror
of the C ABI): single contour steps on device and host buffers, whole SCFT
iterations in both precisions and schemes and every storage mode, batches,
and the warm-start network.  Sizes are those of the repository's own
configurations, tests and benchmark workloads, or lie between them; chains of
the large grids are shortened (every contour step costs the same).

A case is a dict:
  kind   "step" (allocation-free step on device arrays), "driver" (init_pr +
         mde_one_step on host arrays), "scft" (whole iterations), "batch",
         "net" (warm-start network: prediction, loss and gradient)
  n, L, nmax   grid edge, highest harmonic degree, contour steps
  fa, fc       fractions of the A and C blocks
  x            contour / persistence length; box: box edge in radii of gyration
  chi, nmu     interaction parameters; nmu != 0 switches the Maier-Saupe term on
  prec         "fp64" (the drop-in) or "fp32" propagators
  lit          "real4" (literals of a standard Fortran build) or "real8"
  store, ckpt  storage mode (1 all slices, 0 streamed, 2 streamed with the
               orientation tensor) and checkpoint interval
  scheme       "bdf" or "split"
  iters, simple, depth   SCFT iterations of one pass, the simple-mixing ones
               among them, the Anderson depth
Results of the FP32 form carry 32 bits and are handed on in that type.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_REPO, "wormlike-chain-triblock_gb300")

_BASE = dict(kind="scft", n=32, L=6, nmax=40, fa=0.34, fc=0.34, x=2.0, box=5.0, chi=18.0, nmu=0.0, prec="fp64",
             lit="real4", store=1, ckpt=0, scheme="bdf", iters=1, simple=20, depth=5)


def _case(name, **kw):
    return dict(_BASE, name=name, **kw)


def listed():
    return [
        # one contour step inside a caller's own loop, on its device buffers: the smallest call, where latency counts
        _case("step_16_L4", kind="step", n=16, L=4, nmax=10),
        # the step interface a Fortran driver calls (init_pr, mde_one_step) at the CPU reference configuration
        _case("driver_32_L6", kind="driver", n=32, L=6, nmax=100),
        # a short SCFT run on a small grid (parameter scans, training data): launches and small kernels
        _case("scft_16_L2", n=16, L=2, nmax=20, iters=4, simple=2),
        # one iteration of the CPU reference configuration
        _case("scft_32_L6", n=32, L=6, nmax=100, fa=0.33),
        # one iteration of the headline workload (shorter chain), the FP64 drop-in
        _case("scft_64_L10", n=64, L=10, nmax=40, fa=0.25, fc=0.25),
        # the same workload in the FP32 form
        _case("scft_64_L10_fp32", n=64, L=10, nmax=100, fa=0.25, fc=0.25, prec="fp32"),
        # a grid that is no power of two, default-real-8 literals, streamed densities and a checkpointed chain
        _case("stream_48_L8", n=48, L=8, nmax=30, fa=0.27, fc=0.4, store=0, ckpt=10, lit="real8"),
        # the operator-split scheme on an odd-radix grid
        _case("split_40_L7_fp32", n=40, L=7, nmax=64, scheme="split", prec="fp32", x=1.3),
        # liquid-crystalline blocks (Maier-Saupe coupling, orientation tensor) in FP64
        _case("ms_24_L5", n=24, L=5, nmax=30, nmu=3.0, x=4.0),
        # the large workload: 128^3, L=12, Maier-Saupe, FP32, streamed and checkpointed (shorter chain)
        _case("ms_128_L12_fp32", n=128, L=12, nmax=6, box=8.0, chi=20.0, nmu=5.0, x=4.0, prec="fp32", store=2, ckpt=3),
        # parameter sweep: independent instances on mixed grids advanced together
        _case("batch_12", kind="batch", n=48, L=8, nmax=64, prec="fp32", store=0, count=12),
        # the warm start: one prediction, and loss and gradient of one training sample
        _case("net_32", kind="net", n=32, width=32, prec="fp32"),
    ]


def _cost(c):
    """Rough seconds of one pass, to keep drawn cases within the largest listed one."""
    if c["kind"] == "net":
        return 0.01 * (c["n"] / 32.0) ** 3 * (c["width"] / 32.0) ** 2
    M, pts = (c["L"] + 1) ** 2, float(c["n"]) ** 3
    steps = 2.0 * c["nmax"] * c["iters"] if c["kind"] in ("scft", "batch") else 2.0
    per = M * pts * (2.4e-10 if c["prec"] == "fp64" else 2.5e-11)
    if c["nmu"]:
        per *= 3.0
    if c["ckpt"]:
        per *= 1.5
    return steps * (6e-5 + per) * c.get("count", 1)


def _fits(c):
    """Whether the library has this size: a coefficient column in shared memory (its own refusal, WLC_E_UNSUPPORTED)."""
    M, n = (c["L"] + 1) ** 2, c["n"]
    if c["kind"] == "net":
        return True
    if c["kind"] == "step" and M * (n // 2 + 1) * n * n * 16 > 62 * 2 ** 20:
        return False
    if c["prec"] == "fp64":
        if n > 96:
            return False
        return M * ((n + 1) * 16 + (n * 8 + 60 if c["lit"] == "real4" else 0)) < 215e3
    return M * (n + 1) * 8 < 220e3


def draw(rng):
    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    while True:
        c = dict(_BASE)
        c["kind"] = rng.choice(["step", "driver", "scft", "scft", "scft", "scft", "scft", "scft", "batch", "net"])
        if c["kind"] == "net":
            c.update(n=rng.choice([16, 24, 32, 40]), width=rng.choice([16, 32, 48]), prec="fp32")
            return c
        edges = [12, 16, 24, 32, 40, 48, 64, 96, 128]
        c["n"] = min(edges, key=lambda e: abs(math.log(e / log(11, 136))))
        c["L"] = int(round(log(2, 12)))
        c["nmax"] = 2 * int(round(log(8, 60)))
        c["fa"], c["fc"] = round(rng.uniform(0.2, 0.4), 3), round(rng.uniform(0.2, 0.4), 3)
        c["x"] = round(rng.uniform(0.5, 4.0), 2)
        c["box"] = round(rng.uniform(3.5, 8.0), 2)
        c["chi"] = round(rng.uniform(12.0, 24.0), 1)
        c["prec"] = rng.choice(["fp64", "fp32"])
        c["lit"] = rng.choice(["real4", "real4", "real8"])
        if c["kind"] == "step":
            c["prec"] = "fp64"
        elif c["kind"] == "batch":
            c.update(prec="fp32", store=0, count=rng.randint(3, 16))
            c["n"] = rng.choice([24, 32, 40, 48])
        elif c["kind"] == "scft":
            c["store"] = rng.choice([1, 1, 0, 2])
            if c["store"] != 1 and c["nmax"] >= 12 and rng.random() < 0.5:
                c["ckpt"] = int(math.sqrt(3 * c["nmax"]))
            c["scheme"] = rng.choice(["bdf", "bdf", "bdf", "split"])
            if c["scheme"] == "bdf" and rng.random() < 0.35:
                c["nmu"] = round(rng.uniform(2.0, 6.0), 1)
        if _fits(c) and _cost(c) <= 0.4 and c["n"] ** 3 * (c["L"] + 1) ** 2 * (c["nmax"] + 1) <= 2 ** 31:
            return c


# ------------------------------------------------------------------ inputs
def _rg(x):
    return math.sqrt(1.0 / (3.0 * x) - 1.0 / x ** 2 + 2.0 / x ** 3 - 2.0 / x ** 4 * (1.0 - math.exp(-x)))


def _even(v):
    return int(2 * math.floor(v / 2.0 + 0.5))


def _blocks(c):
    na, nc = _even(c["fa"] * c["nmax"]), _even(c["fc"] * c["nmax"])
    return na, c["nmax"] - na - nc, nc


def _members(c):
    """The instances of a case: one, or a batch's, on mixed grids with their own parameters."""
    if c["kind"] != "batch":
        return [dict(c)]
    out = []
    for j in range(c["count"]):
        m = dict(c)
        m["n"] = [c["n"], 24, 32, 40][j % 4]
        m["fa"] = round(0.2 + 0.2 * ((j * 0.37 + c["fa"]) % 1.0), 3)
        m["fc"] = round(0.2 + 0.2 * ((j * 0.61 + c["fc"]) % 1.0), 3)
        m["x"] = round(0.5 + 2.5 * ((j * 0.73 + c["x"] / 8) % 1.0), 2)
        m["chi"] = round(12.0 + 12.0 * ((j * 0.29 + c["chi"] / 24) % 1.0), 1)
        out.append(m)
    return out


def _params(c):
    """make_params arguments: kappa and Loa from contour / persistence, the box edge in radii of gyration."""
    return dict(n=c["n"], lmax=c["L"], nmax=c["nmax"], ns=_blocks(c), dx=c["box"] * _rg(c["x"]) / c["n"],
                loa=0.5 * c["x"], kappa=(0.5, 0.5, 0.5), chi=(c["chi"],) * 3, nmu=c["nmu"],
                precision=0 if c["prec"] == "fp64" else 1, literals=0 if c["lit"] == "real4" else 1,
                store_qstar=c["store"], q_checkpoint=c["ckpt"], scheme=0 if c["scheme"] == "bdf" else 1)


def _fields(c, seed):
    """Block fields half way to an ordered phase (a few long waves of the size of chi about a common level) with noise,
    within what the contour step is stable for, and the Maier-Saupe tensor (symmetric, traceless) of a case that has one."""
    rng = np.random.default_rng([int(seed), c["n"], c["L"]])
    n = c["n"]
    x = 2.0 * np.pi * np.arange(n) / n
    a = min(0.08 * c["chi"], 0.1 * c["nmax"])
    w = np.full((3, n, n, n), 2.5 * a)
    for b in range(3):
        for _ in range(3):
            k = rng.integers(-2, 3, size=3)
            ph = rng.uniform(0, 2 * np.pi)
            w[b] += a * np.cos(k[0] * x[None, None, :] + k[1] * x[None, :, None] + k[2] * x[:, None, None] + ph)
    w = w.reshape(3, -1) + rng.normal(0.0, 0.3, size=(3, n ** 3))
    m = None
    if c["nmu"]:
        a = rng.normal(0.0, 0.2, size=(6, n ** 3))
        m = np.empty((3, 3, n ** 3))
        for q, (i, j) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
            m[i, j] = a[q]
            m[j, i] = a[q]
        tr = (m[0, 0] + m[1, 1] + m[2, 2]) / 3.0
        for i in range(3):
            m[i, i] -= tr
    return w, m


def _slice(c, seed):
    """A right-hand side as the sweeps make it, [coefficient][point]: smooth in space, falling with the degree."""
    g = torch.Generator(device="cpu").manual_seed(int(seed) * 7919 + c["n"] * 31 + c["L"])
    M, n = (c["L"] + 1) ** 2, c["n"]
    deg = torch.tensor([int(math.isqrt(i)) for i in range(M)], dtype=torch.float64)
    a = torch.randn(M, n, n, n, generator=g, dtype=torch.float64)
    a = a + torch.roll(a, 1, 1) + torch.roll(a, 1, 2) + torch.roll(a, 1, 3)
    a = a * (0.5 ** deg)[:, None, None, None]
    a[0] += 1.0
    return a.reshape(M, n ** 3)


def _net_inputs(c, seed):
    rng = np.random.default_rng([int(seed), c["n"], c["width"]])
    P = c["n"] ** 3
    h = c["n"] // 2
    noise = rng.normal(size=(h, h, h)).astype(np.float32).repeat(2, 0).repeat(2, 1).repeat(2, 2)
    x = np.concatenate([noise.reshape(1, P), np.repeat(rng.uniform(-1, 1, size=(5, 1)), P, axis=1)]).astype(np.float32)
    t = rng.normal(0.0, 0.3, size=(3, P)).astype(np.float32)
    return x, t


def _net_shapes(C):
    """(input channels, output channels, stride) of the ten convolutions."""
    return [(16, C, 1), (C, 2 * C, 2), (2 * C, 2 * C, 1), (2 * C, 4 * C, 2), (4 * C, 4 * C, 1), (4 * C, 4 * C, 2),
            (8 * C, 4 * C, 1), (6 * C, 2 * C, 1), (3 * C, C, 1), (C, 16, 1)]


def _net_weights(c, seed):
    """Parameters of a trained network's size: weights ~ N(0, 2 / inputs), small biases, in the library's order."""
    rng = np.random.default_rng([int(seed) + 1, c["width"]])
    out = []
    for ci, co, _ in _net_shapes(c["width"]):
        out.append(rng.normal(0.0, math.sqrt(2.0 / (27 * ci)), size=27 * ci * co))
        out.append(rng.normal(0.0, 0.02, size=co))
    return np.concatenate(out).astype(np.float32)


def _wlc():
    if _PKG not in sys.path:
        sys.path.insert(0, _PKG)
    import wlc
    return wlc


G_INDEX = 4  # third-order step of the B block, forward


def prepare(case, seed):
    wlc = _wlc()
    c = case
    if c["kind"] == "net":
        x, t = _net_inputs(c, seed)
        net = wlc.WarmStartNet(grid=c["n"], width=c["width"])
        net.set_params(_net_weights(c, seed))
        return dict(c=c, net=net, x=x, t=t)
    if c["kind"] == "step":
        f = wlc.load().wlc_mde_one_step_noalloc
        f.argtypes = [ctypes.POINTER(wlc.Params), ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p,
                      ctypes.c_char_p, ctypes.c_int32]
        f.restype = ctypes.c_int
        pr = _slice(c, seed).cuda()
        return dict(c=c, f=f, p=wlc.make_params(**_params(c)), pr=pr, q=torch.empty_like(pr),
                    err=ctypes.create_string_buffer(256))
    if c["kind"] == "batch":
        ms = _members(c)
        b = wlc.Batch([_params(m) for m in ms])
        return dict(c=c, b=b, w=[_fields(m, seed * 100 + j)[0] for j, m in enumerate(ms)])
    inst = wlc.Instance(**_params(c))
    if c["kind"] == "driver":
        inst.set_fields(_fields(c, seed)[0])
        q = np.ascontiguousarray(_slice(c, seed).numpy().T)
        for j in range(3):  # the stored history of contour index s
            inst.set_q(1, _blocks(c)[0] + 1 + j, q * (1.0 - 0.02 * j))
        return dict(c=c, inst=inst)
    w, m = _fields(c, seed)
    mix = wlc.mix_params(anderson_depth=c["depth"], num_simple=c["simple"])
    return dict(c=c, inst=inst, w=w, m=m, mix=mix)


def _typed(c, out):
    """Results in the type the propagators were computed in."""
    if c["prec"] == "fp64":
        return out
    return {k: np.asarray(v, dtype=np.float32) if not isinstance(v, list) else [_typed(c, x) for x in v]
            for k, v in out.items()}


def run(state):
    c = state["c"]
    if c["kind"] == "step":
        rc = state["f"](ctypes.byref(state["p"]), G_INDEX, state["pr"].data_ptr(), state["q"].data_ptr(),
                        torch.cuda.current_stream().cuda_stream, state["err"], 256)
        if rc != 0:
            raise RuntimeError(state["err"].value.decode())
        return state["q"]
    if c["kind"] == "net":
        y = state["net"].forward(state["x"])
        loss, grad = state["net"].loss_grad(state["x"], state["t"])
        return dict(y=y, loss=np.float32(loss), grad=grad)
    if c["kind"] == "driver":
        inst, s = state["inst"], _blocks(c)[0] + 4
        pr = inst.init_pr(1, s)
        return _typed(c, dict(pr=pr, q=inst.mde_one_step(G_INDEX, pr)))
    if c["kind"] == "batch":
        b = state["b"]
        for inst, w in zip(b.instances, state["w"]):
            inst.set_fields(w)
        b.propagate()
        out = []
        for inst in b.instances:
            d = inst.density(want_junction=False)
            out.append(dict(phi=d["phi"], lnQ=d["lnQ"], F=inst.free_energy()))
        return _typed(c, dict(members=out))
    inst = state["inst"]
    inst.set_fields(state["w"], state["m"])
    inst.reset_mixing()
    want_s = bool(c["nmu"]) or c["store"] == 2
    for _ in range(c["iters"]):
        inst.calc_THETAij()
        inst.MDE_q()
        inst.MDE_qstar()
        d = inst.density(want_s=want_s)
        fe = inst.free_energy()
        err, _conv = inst.iterate(state["mix"])
    out = dict(F=fe, lnQ=d["lnQ"], phi=d["phi"], junction=d["junction"], err=err, w=inst.get_fields())
    if want_s:
        out["S"] = d["S"]
    if c["nmu"]:
        out["M"] = inst.get_mop()
    return _typed(c, out)


def work(case):
    c = case
    if c["kind"] == "net":
        # 27 neighbours per channel pair at each level; forward twice, the two gradients once each
        C, P = c["width"], c["n"] ** 3
        shapes, level = _net_shapes(C), [1, 2, 2, 4, 4, 8, 4, 2, 1, 1]  # output grid n / level
        mac = sum(27 * ci * co * P / s ** 3 for (ci, co, _), s in zip(shapes, level))
        par = 27 * sum(ci * co for ci, co, _ in shapes)
        return dict(bytes=8.0 * par + 4.0 * (9 + 3) * P, flops=2.0 * 4 * mac)
    total = dict(bytes=0.0, flops=0.0)
    for m in _members(c):
        M, N, b = (m["L"] + 1) ** 2, m["n"], 8 if m["prec"] == "fp64" else 4
        pts, nk = float(N) ** 3, N * N * (N // 2 + 1)
        rot = sum(l * l + l + 1 for l in range(m["L"] + 1))
        # two real transforms of every coefficient, and per wavevector the factorised solve: the constant rotation
        # and its transpose twice each, four rotations about z, the tridiagonal sweeps (complex by real)
        step = 2 * 2.5 * pts * math.log2(pts) * M + nk * (4 * 4.0 * rot + 4 * 6.0 * M + 8.0 * M)
        if m["kind"] == "step":
            total["bytes"] += 16.0 * M * pts
            total["flops"] += step
        elif m["kind"] == "driver":
            total["bytes"] += 4 * 8.0 * M * pts + 3 * b * M * pts
            total["flops"] += step + 6 * M * pts
        else:
            steps = 2 * m["nmax"] * m["iters"]
            total["bytes"] += steps * (4.0 * b * M * pts + 8 * pts) + 8.0 * 12 * pts * m["iters"]
            total["flops"] += steps * (step + 6 * M * pts) + steps * 2.0 * M * pts
            if m["nmu"]:  # about ten coupled coefficients a row: five products each, and the tensor's five forms
                total["flops"] += steps * pts * M * 10 * 14.0
    return total


# ------------------------------------------------------------------ the same in 64 bits
def _harmonics(L, ct, phi):
    """Real harmonics at points (Condon-Shortley phase in P_l^m; cos for m > 0, sin for m < 0), [M][points]."""
    st = np.sqrt(1.0 - ct * ct)
    P = {(0, 0): np.ones_like(ct)}
    for m in range(1, L + 1):
        P[m, m] = -(2 * m - 1) * st * P[m - 1, m - 1]
    for m in range(L):
        P[m + 1, m] = (2 * m + 1) * ct * P[m, m]
    for m in range(L + 1):
        for l in range(m + 2, L + 1):
            P[l, m] = ((2 * l - 1) * ct * P[l - 1, m] - (l + m - 1) * P[l - 2, m]) / (l - m)
    Y = []
    for l in range(L + 1):
        for m in range(-l, l + 1):
            a = abs(m)
            nrm = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - a) / math.factorial(l + a))
            if m:
                nrm *= math.sqrt(2.0)
            Y.append(nrm * P[l, a] * (1.0 if m == 0 else np.cos(a * phi) if m > 0 else np.sin(a * phi)))
    return np.array(Y)


def _couplings(L, real4):
    """R, T, J: sqrt(4 pi) times the integral of three harmonics, with the square-root factors in the literals' precision."""
    f = np.float32 if real4 else np.float64
    x, wx = np.polynomial.legendre.leggauss(L + 3)
    na = 2 * L + 5
    ph = 2 * np.pi * np.arange(na) / na
    ct, phi, wq = np.repeat(x, na), np.tile(ph, len(x)), np.repeat(wx, na) * 2 * np.pi / na
    Y = _harmonics(max(L, 2), ct, phi)
    M = (L + 1) ** 2
    ls = np.array([math.isqrt(i) for i in range(M)])
    ms = np.arange(M) - ls * ls - ls

    def triple(l3, m3):
        t = math.sqrt(4 * math.pi) * (Y[:M] * (wq * Y[l3 * l3 + l3 + m3])) @ Y[:M].T
        t[np.abs(t) < 1e-13] = 0.0
        P = ((2 * ls[:, None] + 1) * (2 * ls[None, :] + 1) * (2 * l3 + 1)).astype(np.float64)
        root = np.sqrt(P.astype(f)).astype(np.float64)
        neg = (ms[:, None] < 0).astype(int) + (ms[None, :] < 0) + (m3 < 0)
        zero = (ms[:, None] == 0) | (ms[None, :] == 0) | (m3 == 0)
        r = np.where(zero, root / np.sqrt(P), root / float(np.sqrt(f(2.0))) / np.sqrt(P / 2))
        half = np.sqrt((P.astype(f) / f(2.0)).astype(f)).astype(np.float64) / np.sqrt(P / 2)
        return t * np.where(~zero & (neg == 0), half, r)

    def lit(a, b):
        return float(f(a) / np.sqrt(f(b)))

    cR, c15, c5, c215 = lit(1, 3), lit(1, 15), lit(1, 5), lit(2, 15)
    cJ = float(f(-1.0) / (f(3.0) * np.sqrt(f(5.0))))
    R = [-cR * triple(1, 1), -cR * triple(1, -1), cR * triple(1, 0)]
    t22, t20, t2m2, t21, t2m1 = triple(2, 2), triple(2, 0), triple(2, -2), triple(2, 1), triple(2, -1)
    T = [c15 * t22, c5 * t20, c215 * t2m2, -c215 * t21, -c215 * t2m1]
    J = [c15 * t22 + cJ * t20, -c15 * t22 + cJ * t20, c15 * t2m2, -c15 * t21, -c15 * t2m1]
    return R, T, J


class _Exact:
    """One instance in FP64: FFTs by torch, the operator solved degree block by degree block (k.R couples l and l+1
    only, so elimination in l leaves one real symmetric matrix per degree and wavevector)."""

    def __init__(self, c):
        self.c = c
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.N, self.L, self.M, self.nmax = c["n"], c["L"], (c["L"] + 1) ** 2, c["nmax"]
        self.ns = _blocks(c)
        self.start = (0, self.ns[0], self.ns[0] + self.ns[1])
        p = _params(c)
        self.dx, self.loa, self.nr = p["dx"], p["loa"], self.N ** 3
        r4 = self.r4 = c["lit"] == "real4"
        self.ds, self.vol = 1.0 / self.nmax, self.dx ** 3 * self.nr
        self.c0 = {1: 1.0, 2: 1.5, 3: float(np.float32(11.0) / np.float32(6.0)) if r4 else 11.0 / 6.0}
        self.third = float(np.float32(1.0) / np.float32(3.0)) if r4 else 1.0 / 3.0
        self.thresh = float(np.float32(1e-10)) if r4 else 1e-10
        pi2 = float(np.float32(2.0) * np.float32(3.14159265358979323846)) if r4 else 2.0 * math.pi
        R, T, J = _couplings(self.L, r4)
        self.R = [self.t(a) for a in R]
        self.T, self.J = torch.stack([self.t(a) for a in T]), [self.t(a) for a in J]
        k = np.arange(self.N)
        k = np.where(k <= self.N // 2, k, k - self.N) * (pi2 / (self.N * self.dx))
        k = self.t(k)
        nkx = self.N // 2 + 1
        z, y, x = torch.meshgrid(k, k, k[:nkx], indexing="ij")
        self.k = [x.reshape(-1), y.reshape(-1), z.reshape(-1)]
        self.cache = {}
        s = self.t(np.where(np.arange(self.N) % 2, 4.0, 2.0) * self.dx / 3.0)
        self.w3 = (s[:, None, None] * s[None, :, None] * s[None, None, :]).reshape(-1)

    def t(self, a):
        return torch.as_tensor(np.asarray(a, dtype=np.float64), device=self.dev)

    def sl(self, l):
        return slice(l * l, (l + 1) * (l + 1))

    def coupling(self, l, ds):  # ds k.R between degrees l and l+1: [nk][2l+1][2l+3] and its partner
        up = sum(self.k[a][:, None, None] * (ds * self.R[a][self.sl(l), self.sl(l + 1)]) for a in range(3))
        dn = sum(self.k[a][:, None, None] * (ds * self.R[a][self.sl(l + 1), self.sl(l)]) for a in range(3))
        return up, dn

    def solve(self, b, c0, ds, sigma):
        """G x = b, b complex [nk][M]; G = c0 + ds Loa l(l+1)/(2 kappa) + i sigma ds k.R, kappa = 1/2 in every block."""
        key = (c0, ds)
        if key not in self.cache:
            inv, cpl = [], []
            for l in range(self.L + 1):
                a = c0 + ds * self.loa * l * (l + 1)
                D = torch.eye(2 * l + 1, device=self.dev, dtype=torch.float64).expand(b.shape[0], -1, -1) * a
                if l:
                    D = D + cpl[l - 1][1] @ inv[l - 1] @ cpl[l - 1][0]
                inv.append(torch.linalg.inv(D))
                if l < self.L:
                    cpl.append(self.coupling(l, ds))
            self.cache = {key: (inv, cpl)} if self.N > 48 and len(self.cache) > 2 else {**self.cache, key: (inv, cpl)}
        inv, cpl = self.cache[key]
        v = torch.view_as_real(b.contiguous())

        def times_i(u, f):
            return f * torch.stack([-u[..., 1], u[..., 0]], dim=-1)

        y = [None] * (self.L + 1)
        for l in range(self.L + 1):
            y[l] = v[:, self.sl(l)]
            if l:
                y[l] = y[l] - times_i(cpl[l - 1][1] @ y[l - 1], sigma)
            y[l] = y[l].contiguous()
            if l < self.L:
                y[l] = inv[l] @ y[l]  # D^-1 y, which the next degree and the way back both want
        x = [None] * (self.L + 1)
        x[self.L] = inv[self.L] @ y[self.L]
        for l in range(self.L - 1, -1, -1):
            x[l] = y[l] - inv[l] @ times_i(cpl[l][0] @ x[l + 1], sigma)
        return torch.view_as_complex(torch.cat(x, dim=1).contiguous())

    def transform(self, pr, op):
        """C2R(op(R2C(pr)))/N^3 of [M][nr]; the imaginary parts at kx = 0 and N/2 are dropped before the last transform."""
        n = self.N
        f = torch.fft.rfftn(pr.reshape(self.M, n, n, n), dim=(1, 2, 3))
        f = op(f.reshape(self.M, -1).T).T.reshape(f.shape)
        f = torch.fft.ifftn(f, dim=(1, 2))
        f[..., 0].imag.zero_()
        f[..., n // 2].imag.zero_()
        return torch.fft.irfft(f, n=n, dim=3).reshape(self.M, -1)

    def one_step(self, pr, order, sigma):
        return self.transform(pr, lambda b: self.solve(b, self.c0[order], self.ds, sigma))

    def rhs(self, h, w, order):
        ds, W = self.ds, w[None, :]
        if order == 1:
            hh = h[0]
            pr = (1.0 - ds * W) * h[0]
        elif order == 2:
            hh = 2 * h[0] - h[1]
            pr = 2 * h[0] - 0.5 * h[1] - ds * W * hh
        else:
            hh = 3 * h[0] - 3 * h[1] + h[2]
            pr = (3 - 3 * ds * W) * h[0] + (-1.5 + 3 * ds * W) * h[1] + (self.third - ds * W) * h[2]
        if self.theta is not None:
            pr = pr + ds * torch.bmm(self.theta, hh.T.unsqueeze(2)).squeeze(2).T
        return pr

    def step(self, h, blk, order, sigma):
        if self.c["scheme"] == "split":
            e = torch.exp(-0.5 * self.ds * self.w[blk])[None, :]
            return e * self.transform(e * h[0], lambda b: 2 * self.solve(b, 1.0, 0.5 * self.ds, sigma) - b)
        return self.one_step(self.rhs(h, self.w[blk], order), order, sigma)

    def set_fields(self, w, m):
        self.w = w
        self.m = m
        self.theta = None
        if m is not None:
            co = torch.stack([m[0] - m[4], m[8], m[3], m[6], m[7]])
            self.theta = torch.einsum("cr,cij->rij", co, self.T)
            self.theta[self.theta.abs() < self.thresh] = 0.0

    def sweeps(self):
        q = [torch.zeros(self.M, self.nr, device=self.dev, dtype=torch.float64)]
        q[0][0] = 1.0
        for s in range(1, self.nmax + 1):
            blk = 0 if s <= self.start[1] else 1 if s <= self.start[2] else 2
            q.append(self.step([q[s - j] for j in (1, 2, 3) if s >= j], blk, min(s, 3), 1))
        raw = torch.zeros(3, self.nr, device=self.dev, dtype=torch.float64)
        sraw = torch.zeros(3, 5, self.nr, device=self.dev, dtype=torch.float64)
        junc = torch.zeros(3, self.nr, device=self.dev, dtype=torch.float64)
        p = [q[0].clone()]
        for i in range(self.nmax + 1):
            s = self.nmax - i
            if i:
                blk = 2 if s >= self.start[2] else 1 if s >= self.start[1] else 0
                p.insert(0, self.step(p[:3], blk, min(i, 3), -1))
                del p[3:]
            dot = (q[s] * p[0]).sum(0)
            form = [(q[s] * (J @ p[0])).sum(0) for J in self.J] if self.want_s else []
            for b in range(3):
                j = s - self.start[b]
                if self.ns[b] > 0 and 0 <= j <= self.ns[b]:
                    wt = (1.0 if j in (0, self.ns[b]) else 4.0 if j % 2 else 2.0) * self.ds / 3.0
                    raw[b] += wt * dot
                    for a, v in enumerate(form):
                        sraw[b, a] += wt * v
            for a, sj in enumerate((self.start[1], self.start[2], self.nmax)):
                if s == sj:
                    junc[a] = dot
        return raw, sraw, junc, q[self.nmax][0]

    def s3(self, a):
        return float((self.w3 * a).sum())

    def density(self):
        raw, sraw, junc, qend = self.sweeps()
        f = self.vol / self.s3(raw.sum(0))
        self.phi, self.junc = raw * f, junc * f
        self.lnq = math.log(self.s3(qend) / self.vol)
        sx = sraw * f
        xx, yy, xy, xz, yz = (sx[:, a] for a in range(5))
        self.S = torch.stack([xx, xy, xz, xy, yy, yz, xz, yz, -(xx + yy)], dim=1)

    def free_energy(self):
        p, w, chi = self.phi, self.w, self.c["chi"]
        v = chi * (p[0] * p[1] + p[0] * p[2] + p[1] * p[2]) - (w * p).sum(0) + w.sum(0) / 3.0 * (p.sum(0) - 1.0)
        if self.m is not None:
            m = self.m.reshape(3, 3, -1)
            v = v + 0.5 * (m * m.transpose(0, 1)).sum((0, 1)) / self.c["nmu"]
        return -self.lnq + self.s3(v) / self.vol

    def dot(self, a, b):
        return self.s3((a * b).sum(0) if a.dim() > 1 else a * b) / self.vol

    def mix(self, it, hist):
        """iterate(): simple mixing, then Anderson with the history in the order of the iterations."""
        c, phi, w = self.c, self.phi, self.w
        C = torch.full((3, 3), c["chi"], device=self.dev, dtype=torch.float64)
        C.fill_diagonal_(0.0)
        f = self.t(self.ns) / self.nmax
        err = np.zeros(5)
        err[3] = float((phi.sum(0) - 1.0).abs().max())
        wout = C @ phi + (w.sum(0) - (C @ f).sum()) / 3.0
        if it >= c["simple"]:
            hist.insert(0, (wout, wout - w))
            del hist[c["depth"] + 1:]
        if it <= c["simple"]:
            dw = C @ (phi - f[:, None]) + w.sum(0) / 3.0 - w
            new = w + 0.1 * dw
            err[:3] = dw.abs().amax(1).cpu().numpy()
        else:
            (wk, dk), old = hist[0], hist[1:]
            e = [dk - d for _, d in old]
            U = np.array([[self.dot(a, b) for b in e] for a in e])
            V = np.array([self.dot(a, dk) for a in e])
            co = np.linalg.solve(U, V)
            wi = wk + sum(float(a) * (ww - wk) for a, (ww, _) in zip(co, old))
            di = dk + sum(float(a) * (d - dk) for a, (_, d) in zip(co, old))
            new = wi + 0.1 * di
            for b in range(3):
                err[b] = math.sqrt(abs(self.dot(dk[b], dk[b]) / self.dot(wk[b], wk[b])))
        m = self.m
        if m is not None:
            d = c["nmu"] * self.S.sum(0) - m
            m = m + 0.08 * d
            err[4] = float(d.abs().max())
        self.set_fields(new, m)
        return err

    def run(self, w, m):
        self.want_s = bool(self.c["nmu"]) or self.c["store"] == 2
        self.set_fields(self.t(w), None if m is None else self.t(m.reshape(9, -1)))
        hist = []
        for it in range(1, self.c["iters"] + 1):
            self.density()
            fe = self.free_energy()
            err = self.mix(it, hist)
        n = self.nr
        out = dict(F=fe, lnQ=self.lnq, phi=self.phi, junction=self.junc, err=err, w=self.w)
        if self.want_s:
            out["S"] = self.S.reshape(3, 3, 3, n)
        if self.c["nmu"]:
            out["M"] = self.m.reshape(3, 3, n)
        return {k: v.cpu().numpy() if isinstance(v, torch.Tensor) else v for k, v in out.items()}


def _exact_net(c, seed):
    """The network in 64 bits (no BF16 anywhere): torch's convolutions and its gradient, in the library's layouts."""
    import torch.nn.functional as F
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, t = _net_inputs(c, seed)
    flat = torch.as_tensor(_net_weights(c, seed).astype(np.float64), device=dev).requires_grad_(True)
    n, shapes = c["n"], _net_shapes(c["width"])
    off = [0]

    def conv(i, v):
        ci, co, s = shapes[i]
        w = flat[off[0]:off[0] + 27 * ci * co].reshape(3, 3, 3, ci, co).permute(4, 3, 0, 1, 2)
        b = flat[off[0] + 27 * ci * co:off[0] + 27 * ci * co + co]
        off[0] += 27 * ci * co + co
        # one neighbour at a time: torch has no fast 64-bit convolution
        g = v.shape[-1] // s
        y = b[:, None].expand(co, g ** 3)
        for k in range(27):
            d = (k // 9 - 1, k // 3 % 3 - 1, k % 3 - 1)
            u = torch.roll(v, (-d[0], -d[1], -d[2]), (1, 2, 3))[:, ::s, ::s, ::s].reshape(ci, -1)
            y = y + w[:, :, k // 9, k // 3 % 3, k % 3] @ u
        y = y.reshape(co, g, g, g)
        return y if i == 9 else F.relu(y)

    def up(v):
        return v.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    v = torch.zeros(16, n, n, n, device=dev, dtype=torch.float64)
    v[:6] = torch.as_tensor(x.astype(np.float64), device=dev).reshape(6, n, n, n)
    e1 = conv(0, v)
    e2 = conv(1, e1)
    e3 = conv(2, e2)
    e5 = conv(4, conv(3, e3))
    d1 = conv(6, torch.cat([up(conv(5, e5)), e5]))
    d2 = conv(7, torch.cat([up(d1), e3]))
    y = conv(9, conv(8, torch.cat([up(d2), e1])))[:3].reshape(3, -1)
    loss = ((y - torch.as_tensor(t.astype(np.float64), device=dev)) ** 2).mean()
    loss.backward()
    return dict(y=y.detach().cpu().numpy(), loss=float(loss.detach()), grad=flat.grad.cpu().numpy())


def exact(case, seed):
    c = case
    if c["kind"] == "net":
        return _exact_net(c, seed)
    M, pts = (c["L"] + 1) ** 2, c["n"] ** 3
    if c["nmu"] and pts * M * M > 2 ** 28 or pts * M > 2 ** 25.5:
        return None  # the dense couplings per point, or the blocks per wavevector, would take too long
    if c["kind"] == "step":
        e = _Exact(c)
        return e.one_step(e.t(_slice(c, seed).numpy()), 3, 1).cpu().numpy()
    if c["kind"] == "driver":
        e = _Exact(c)
        w = e.t(_fields(c, seed)[0])
        e.set_fields(w, None)
        a = e.t(_slice(c, seed).numpy())
        s = e.start[1] + 4
        pr = e.rhs([a * (1.0 - 0.02 * j) for j in (2, 1, 0)], w[1 if s <= e.start[2] else 2], 3)
        return dict(pr=pr.T.cpu().numpy(), q=e.one_step(pr, 3, 1).T.cpu().numpy())
    if c["kind"] == "batch":
        out = []
        for j, m in enumerate(_members(c)):
            e = _Exact(m)
            r = e.run(_fields(m, seed * 100 + j)[0], None)
            out.append(dict(phi=r["phi"], lnQ=r["lnQ"], F=r["F"]))
        return dict(members=out)
    return _Exact(c).run(*_fields(c, seed))
