"""Timing cases of the particle-mesh library: the calls a simulation program makes.

Each case goes through the Python mirror of the C ABI (`djb200`) with arrays on the GPU,
or with host arrays where the case says so. Particle states are made from the seed alone:
a Gaussian displacement field (Zel'dovich, a power-law spectrum) and, for late times,
collapsed clumps on top of it. `exact` restates every case in float64 torch.

Kinds
  force       `PMSolver.acceleration(psi)`: one PM force.
  run         `set_state`, `run` over `steps` steps, `get_state`: the body of `run_nbody`.
  hostrun     the same from host arrays to host arrays (`set_state`, `run`, `output`), as
              `run_nbody` does for a caller that holds numpy arrays.
  vjp         `PMSolver.acceleration_vjp(psi, acc_bar)`: the adjoint of one force.
  stepvjp     `PMSolver.step_vjp`: the adjoint of one step.
  pk          `set_state`, `state_power_spectrum`: the snapshot measurement.
  netforward  `ForceNet.apply(x)`: the force-correction network on a mesh.
  netgrads    `ForceNet.backward(x, target)`, `grads()`: the gradients of one training pair.
  corrected   `run` with the network attached: the network-corrected 1x-mesh step.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "discodj.jl_b200"))

DEV = "cuda:0"
NN_HIDDEN, NN_LAYERS, NN_IN, NN_OUT = 32, 4, 4, 3
NN_SCALES = dict(delta_scale=0.2, force_scale=0.15, out_scale=0.02)
PK_BINS = 32


def _case(name, kind, n, res, L=None, W=2, grad=4, aa=0, lap=0, deconv=False, resample=1, late=True, steps=1,
          hidden=NN_HIDDEN):
    return dict(name=name, kind=kind, n=n, res=res, L=float(L if L else 2.0 * n), W=W, grad=grad, aa=aa, lap=lap,
                deconv=deconv, resample=resample, late=late, steps=steps, hidden=hidden)


def listed():
    return [
        # the smallest force a program asks for: the parity-size box, where launches and latency count
        _case("force_cic_64_128", "force", 64, 128, L=250, W=2, grad=2),
        # a whole small run from host arrays to host arrays (64^3 particles, 10 steps to a = 1)
        _case("hostrun_cic_64_128", "hostrun", 64, 128, L=250, W=2, grad=4, late=False, steps=10),
        # a mesh that is no power of two nor a multiple of the bricks, all eight interlacing shifts
        _case("force_tsc_odd_90_180", "force", 90, 180, L=150, W=3, grad=4, aa=2, lap=4, deconv=True),
        # the discreteness-suppressing options of the BullFrog initial conditions: ik gradient,
        # interlacing, 2^3 Fourier sheet resampling
        _case("force_ics_pcs_ik_96_192", "force", 96, 192, L=192, W=4, grad=0, aa=1, deconv=True, resample=2,
              late=False),
        # one step of the 256^3 / 512^3 FastPM configuration: TSC, interlaced, fourth order, late times
        _case("step_tsc_256_512", "run", 256, 512, L=500, W=3, grad=4, aa=1, lap=4),
        # the throughput configuration at 512^3 / 1024^3: PCS, interlaced, sixth order, late times
        _case("step_pcs_512_1024", "run", 512, 1024, L=1000, W=4, grad=6, aa=1),
        # adjoint of the force, as gradient-based inference calls it once per step
        _case("vjp_pcs_256_512", "vjp", 256, 512, L=500, W=4, grad=6, aa=1),
        # adjoint of a step in the differentiable 128^3 / 256^3 CIC run
        _case("stepvjp_cic_128_256", "stepvjp", 128, 256, L=250, W=2, grad=2),
        # P(k) of a resident state
        _case("pk_256_256", "pk", 256, 256, L=500, W=2),
        # the force-correction network: forward on a 256^3 mesh, gradients of one 96^3 pair
        _case("netforward_256", "netforward", 0, 256),
        _case("netgrads_96", "netgrads", 0, 96),
        # one step of the network-corrected run on the 1x mesh: TSC, deconvolved
        _case("corrected_tsc_256_256", "corrected", 256, 256, L=500, W=3, grad=4, deconv=True),
    ]


def _smooth_even(lo, hi):
    """Even sizes in [lo, hi] whose prime factors are at most 7 (what programs choose for transforms)."""
    out = []
    for v in range(lo + lo % 2, hi + 1, 2):
        r = v
        for f in (2, 3, 5, 7):
            while r % f == 0:
                r //= f
        if r == 1:
            out.append(v)
    return out


def _log_pick(rng, sizes):
    target = math.exp(rng.uniform(math.log(sizes[0]), math.log(sizes[-1])))
    return min(sizes, key=lambda v: abs(math.log(v / target)))


def draw(rng):
    kind = rng.choice(["force", "force", "run", "run", "hostrun", "vjp", "stepvjp", "pk", "netforward", "netgrads",
                       "corrected"])
    W, grad = rng.choice([2, 3, 4]), rng.choice([2, 4, 6])
    late = rng.random() < 0.7
    if kind in ("force", "run"):
        res = _log_pick(rng, _smooth_even(48, 640))
        n = max(16, int(res * rng.choice([0.5, 0.5, 1.0, rng.uniform(0.4, 1.0)])))
        n = min(n, 400)
        aa = rng.choice([0, 1, 1, -1, 2] if res <= 320 else [0, 1])
        return _case("", kind, n, res, W=W, grad=grad, aa=aa, lap=rng.choice([0, 0, 2, 4, 6]),
                     deconv=rng.random() < 0.4, late=late, steps=rng.choice([1, 2, 3]) if res <= 320 else 1)
    if kind == "hostrun":
        res = _log_pick(rng, _smooth_even(48, 160))
        return _case("", kind, res // 2, res, W=W, grad=grad, aa=rng.choice([0, 1]), late=False,
                     steps=rng.randint(2, 8))
    if kind in ("vjp", "stepvjp"):
        res = _log_pick(rng, _smooth_even(48, 400))
        n = max(16, int(res * rng.uniform(0.45, 0.9)))
        return _case("", kind, n, res, W=W, grad=grad, aa=rng.choice([0, 1]), late=late)
    if kind == "pk":
        res = _log_pick(rng, _smooth_even(48, 400))
        return _case("", kind, max(16, int(res * rng.uniform(0.5, 1.0))), res, late=late)
    if kind == "netforward":
        return _case("", kind, 0, rng.randint(20, 250))
    if kind == "netgrads":
        return _case("", kind, 0, rng.randint(20, 96))
    res = _log_pick(rng, [v for v in _smooth_even(48, 224) if v % 4 == 0])
    return _case("", kind, max(16, int(res * rng.choice([1.0, rng.uniform(0.5, 1.0)]))), res, W=W, grad=grad,
                 aa=rng.choice([0, 1]), deconv=True, late=late)


# ── inputs ───────────────────────────────────────────────────────────────────
def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed(1_000_003 * int(seed) + salt)


def _wavenumbers(n, L, dtype):
    """(kz, ky, kx) broadcastable to the half spectrum [z][y][x] of an n^3 field."""
    kf = (torch.fft.fftfreq(n, device=DEV, dtype=torch.float64) * n * (2 * math.pi / L)).to(dtype)
    kh = torch.arange(n // 2 + 1, device=DEV, dtype=torch.float64).to(dtype) * (2 * math.pi / L)
    return kf.view(n, 1, 1), kf.view(1, n, 1), kh.view(1, 1, -1)


def _displacements(case, seed):
    """(psi, mom): (3,n,n,n) float32 [c][k][j][i]. Early: a smooth Zel'dovich field of
    r.m.s. contrast 0.03 at growth
    factor 0.02. Late: contrast 1.2 on the lattice scale, and an eighth of the
    8^3-particle Lagrangian blocks contracted to a few cells (collapsed objects)."""
    n, L = case["n"], case["L"]
    white = torch.randn((n, n, n), generator=_gen(seed, 1), device=DEV)
    f = torch.fft.rfftn(white)
    del white
    kz, ky, kx = _wavenumbers(n, L, torch.float32)
    k2 = kx * kx + ky * ky + kz * kz
    k2[0, 0, 0] = 1.0
    knyq = math.pi * n / L
    f *= k2 ** (-0.375) * torch.exp(-k2 / (0.6 * knyq) ** 2)   # P(k) ~ k^-1.5, smoothed at the lattice scale
    f[0, 0, 0] = 0.0
    delta = torch.fft.irfftn(f, s=(n, n, n))
    f *= (1.2 if case["late"] else 0.03) / float(delta.std())
    del delta
    f /= k2
    psi = torch.empty((3, n, n, n), device=DEV)
    for c, k in enumerate((kx, ky, kz)):
        kk = k.clone()
        if n % 2 == 0:
            kk[kk.abs() > knyq * (1 - 1e-6)] = 0.0
        psi[c] = torch.fft.irfftn(1j * kk * f, s=(n, n, n))
    del f, k2
    mom = psi * (0.8 if case["late"] else 50.0)   # early: the growing mode at D = 0.02
    if case["late"]:
        nb = (n + 7) // 8
        hit = torch.rand((nb, nb, nb), generator=_gen(seed, 2), device=DEV) < 0.125
        at = torch.arange(n, device=DEV)
        inside = hit[(at // 8).view(n, 1, 1), (at // 8).view(1, n, 1), (at // 8).view(1, 1, n)]
        off = (at % 8).float() * (L / n) - 3.5 * (L / n)
        for c, shape in enumerate(((1, 1, n), (1, n, 1), (n, 1, 1))):
            psi[c] -= inside * (0.8 * off.view(shape))
        mom += torch.randn((3, n, n, n), generator=_gen(seed, 3), device=DEV) * (0.1 * L / n)
    return psi.contiguous(), mom.contiguous()


def _coefficients(case):
    """FastPM coefficients of an Einstein-de Sitter run (drifts in the growth factor): from
    D = 0.02 to 1 for an early state, a short interval at D = 1 for a late one."""
    d0, d1 = (1.0, 1.0 + 0.05 * case["steps"]) if case["late"] else (0.02, 0.1 if case["steps"] == 1 else 1.0)
    edge = [d0 + (d1 - d0) * i / case["steps"] for i in range(case["steps"] + 1)]
    out = [[], [], [], []]
    for a, b in zip(edge[:-1], edge[1:]):
        m = 0.5 * (a + b)
        alpha = (a / b) ** 1.5
        for v, x in zip(out, (m - a, alpha, (1 - alpha) / m, b - m)):
            v.append(x)
    return out


def _net_layout(case):
    pad = lambda c: (c + 7) // 8 * 8  # noqa: E731
    h = case["hidden"]
    for l in range(NN_LAYERS):
        ci, co = (NN_IN if l == 0 else h), (NN_OUT if l == NN_LAYERS - 1 else h)
        yield ci, co, pad(ci), pad(co)


def _net_params(case, seed):
    """Weights of the usual variance 2/fan-in and small biases, in the library's layout:
    per layer [27 taps][cin padded][cout padded], then the biases; padding entries zero."""
    g = torch.Generator().manual_seed(77 + int(seed))
    parts = []
    for ci, co, cp, op in _net_layout(case):
        w = torch.zeros((27, cp, op))
        w[:, :ci, :co] = torch.randn((27, ci, co), generator=g) * math.sqrt(2.0 / (27 * ci))
        b = torch.zeros(op)
        b[:co] = 0.05 * torch.randn(co, generator=g)
        parts += [w.reshape(-1), b]
    return torch.cat(parts)


def _net_meshes(case, seed):
    r = case["res"]
    x = torch.randn((NN_IN, r, r, r), generator=_gen(seed, 5), device=DEV)
    t = torch.randn((NN_OUT, r, r, r), generator=_gen(seed, 6), device=DEV)
    return x, t


def prepare(case, seed):
    import djb200
    from djb200.nn import ForceNet
    kind = case["kind"]
    st = dict(kind=kind)
    if kind in ("netforward", "netgrads", "corrected"):
        st["net"] = ForceNet(layers=NN_LAYERS, cin=NN_IN, hidden=case["hidden"], cout=NN_OUT)
        st["net"].load(_net_params(case, seed).numpy())
    if kind in ("netforward", "netgrads"):
        st["x"], st["t"] = _net_meshes(case, seed)
        return st
    cfg = djb200.PMConfig(res_pm=case["res"], n_part=case["n"], boxsize=case["L"], worder=case["W"],
                          deconvolve=case["deconv"], antialias=case["aa"], grad_order=case["grad"],
                          lap_order=case["lap"], n_resample=case["resample"])
    st["S"] = djb200.PMSolver(cfg)
    st["psi"], st["mom"] = _displacements(case, seed)
    st["coef"] = _coefficients(case)
    if kind == "corrected":
        st["S"].attach_nn(st["net"], **NN_SCALES)
    if kind == "hostrun":
        st["psi"] = np.asfortranarray(st["psi"].cpu().numpy().transpose(3, 2, 1, 0))
        st["mom"] = np.asfortranarray(st["mom"].cpu().numpy().transpose(3, 2, 1, 0))
    if kind in ("vjp", "stepvjp"):
        st["bar"], st["bar2"] = _cotangents(case, seed)
    return st


def _cotangents(case, seed):
    n = case["n"]
    return (torch.randn((3, n, n, n), generator=_gen(seed, 7), device=DEV),
            torch.randn((3, n, n, n), generator=_gen(seed, 8), device=DEV))


def run(st):
    kind, S = st["kind"], st.get("S")
    if kind == "force":
        return S.acceleration(st["psi"])
    if kind in ("run", "corrected"):
        S.set_state(st["psi"], st["mom"])
        S.run(*st["coef"])
        return S.get_state(device=True)
    if kind == "hostrun":
        S.set_state(st["psi"], st["mom"])
        S.run(*st["coef"])
        return S.output(wrap=0)
    if kind == "vjp":
        return S.acceleration_vjp(st["psi"], st["bar"])
    if kind == "stepvjp":
        return S.step_vjp(*[c[0] for c in st["coef"]], st["psi"], st["mom"], st["bar"], st["bar2"])
    if kind == "pk":
        S.set_state(st["psi"], st["mom"])
        return S.state_power_spectrum(bins=PK_BINS)
    if kind == "netforward":
        return st["net"].apply(st["x"])
    loss = st["net"].backward(st["x"], st["t"])
    return loss, st["net"].grads()


# ── what a pass cannot do without ────────────────────────────────────────────
def _nshift(case):
    return {-1: 1, 0: 1, 1: 2, 2: 8, 3: 16}[case["aa"]]


def _net_flops(case):
    return sum(2 * 27 * ci * co for ci, co, _, _ in _net_layout(case)) * case["res"] ** 3


def work(case):
    """Particle and mesh arrays moved once: a force reads and writes 12 bytes per particle,
    and per shift a density and a potential mesh are each written and read once."""
    kind, nm, npart = case["kind"], case["res"] ** 3, case["n"] ** 3
    nodes = case["W"] ** 3
    if kind == "netforward":
        return dict(bytes=4 * nm * (NN_IN + NN_OUT), flops=_net_flops(case))
    if kind == "netgrads":
        return dict(bytes=4 * nm * (NN_IN + NN_OUT), flops=3 * _net_flops(case))
    fft = 2 * 2.5 * nm * math.log2(nm)
    if kind == "pk":
        return dict(bytes=12 * npart + 8 * nm, flops=fft / 2 + 30 * npart)
    ns, sets = _nshift(case), case["resample"] ** 3
    fields = 3 if case["grad"] == 0 else 1
    one_b = ns * (8 + 8 * fields) * nm + 24 * npart
    one_f = ns * (fft * (1 + fields) / 2 + (sets * 3 + 6 + case["grad"] * 3) * nodes * npart)
    if kind == "force":
        return dict(bytes=one_b, flops=one_f)
    if kind in ("vjp", "stepvjp"):
        extra = 12 if kind == "vjp" else 48
        return dict(bytes=2 * one_b + ns * 24 * nm + extra * npart, flops=2 * one_f + ns * 24 * nodes * npart)
    steps = case["steps"]
    out = dict(bytes=steps * (one_b + 24 * npart), flops=steps * one_f)
    if kind == "corrected":
        out["bytes"] += steps * 28 * nm
        out["flops"] += steps * _net_flops(case)
    return out


def tolerance(case):
    """Positions carry a float32 unit in the last place of the box side, and a force is a
    float32 transform of them; deconvolution and the sharper gradients amplify both."""
    kind = case["kind"]
    if kind in ("netforward", "netgrads"):
        return dict(rel=1e-2, max=0.3)     # bf16 operands and hidden activations
    if kind == "pk":
        return dict(rel=1e-6, max=1e-5)
    if kind in ("vjp", "stepvjp"):
        # the derivative of the piecewise linear CIC weight jumps at cell faces: a particle a
        # rounding away from one may take either side
        return dict(rel=4e-3, max=0.9) if case["W"] == 2 else dict(rel=6e-5, max=1e-2)
    if kind in ("run", "corrected") and case["late"]:
        return dict(rel=4e-6, max=4e-4)    # one or a few kicks on top of the given momenta
    if kind == "force" and (case["grad"] == 0 or case["deconv"]):
        return dict(rel=2e-4, max=4e-3)
    return dict(rel=6e-5, max=4e-3)


# ── float64 restatement ──────────────────────────────────────────────────────
CHUNK = 1 << 22   # particles per pass of the restatement


def _w64(W, d):
    if W == 2:
        return (1 - d).clamp_min(0)
    if W == 3:
        return torch.where(d > 0.5, 0.5 * (1.5 - d).clamp_min(0) ** 2, 0.75 - d * d)
    return torch.where(d > 1, (2 - d).clamp_min(0) ** 3 / 6, 2.0 / 3 - d * d * (1 - 0.5 * d))


def _dw64(W, x):
    """dW/dg at g - node = x."""
    d, s = x.abs(), torch.sign(x)
    if W == 2:
        return -s
    if W == 3:
        return torch.where(d > 0.5, -s * (1.5 - d).clamp_min(0), -2 * x)
    return torch.where(d > 1, -s * 0.5 * (2 - d).clamp_min(0) ** 2, x * (1.5 * d - 2))


class _PM64:
    """The PM force, its pieces and its adjoint in float64 (native [c][z][y][x] arrays)."""

    def __init__(self, case):
        self.c = case
        self.n, self.res, self.L, self.W = case["n"], case["res"], case["L"], case["W"]
        h = 0.5 * self.L / self.res
        z2 = [(a, b, c) for a in (0, h) for b in (0, h) for c in (0, h)]
        self.shifts = {0: [(0, 0, 0)], -1: [(h, h, h)], 1: [(0, 0, 0), (h, h, h)], 2: z2}[case["aa"]]

    def positions(self, psi):
        n = self.n
        X = psi.double().clone()
        q = torch.arange(n, device=psi.device, dtype=torch.float64) * (self.L / n)
        X[0] += q.view(1, 1, n)
        X[1] += q.view(1, n, 1)
        X[2] += q.view(n, 1, 1)
        return X.reshape(3, -1)

    def stencil(self, X, s, W, deriv=False):
        """Per axis: weights (W, m), node indices (W, m) and weight derivatives d/dX."""
        res, L = self.res, self.L
        out = []
        for a in range(3):
            g = torch.remainder(X[a] + s[a], L) / L * res
            b = (torch.floor(g) if W % 2 == 0 else torch.round(g)).long()
            lo = 0 if W == 2 else -1
            w, idx, dw = [], [], []
            for o in range(lo, lo + W):
                x = g - (b + o)
                w.append(_w64(W, x.abs()))
                idx.append(torch.remainder(b + o, res))
                if deriv:
                    dw.append(_dw64(W, x) * (res / L))
            out.append((w, idx, dw))
        return out

    def pieces(self, X, s, W, deriv=False):
        for i in range(0, X.shape[1], CHUNK):
            sl = slice(i, min(i + CHUNK, X.shape[1]))
            yield sl, self.stencil(X[:, sl], s, W, deriv)

    def deposit(self, X, s, W, weight=None):
        res = self.res
        mesh = torch.zeros(res ** 3, dtype=torch.float64, device=X.device)
        for sl, ((wx, ix, _), (wy, iy, _), (wz, iz, _)) in self.pieces(X, s, W):
            for c in range(W):
                for b in range(W):
                    wyz, row = wz[c] * wy[b], (iz[c] * res + iy[b]) * res
                    if weight is not None:
                        wyz = wyz * weight[sl]
                    for a in range(W):
                        mesh.index_add_(0, row + ix[a], wyz * wx[a])
        return mesh.view(res, res, res)

    def gather(self, fields, X, s, W):
        res = self.res
        out = torch.zeros((len(fields), X.shape[1]), dtype=torch.float64, device=X.device)
        for sl, ((wx, ix, _), (wy, iy, _), (wz, iz, _)) in self.pieces(X, s, W):
            for c in range(W):
                for b in range(W):
                    wyz, row = wz[c] * wy[b], (iz[c] * res + iy[b]) * res
                    for a in range(W):
                        idx, w = row + ix[a], wyz * wx[a]
                        for f, field in enumerate(fields):
                            out[f, sl] += field.reshape(-1)[idx] * w
        return out

    def gather_grad(self, fields, coef, X, s, W):
        """(3, Np): sum over fields of coef_f(p) sum_n dW/dX_a field_f(n)."""
        res = self.res
        out = torch.zeros((3, X.shape[1]), dtype=torch.float64, device=X.device)
        for sl, ((wx, ix, dx), (wy, iy, dy), (wz, iz, dz)) in self.pieces(X, s, W, True):
            for c in range(W):
                for b in range(W):
                    row = (iz[c] * res + iy[b]) * res
                    for a in range(W):
                        v = 0
                        for field, co in zip(fields, coef):
                            t = field.reshape(-1)[row + ix[a]]
                            v = v + (t if co is None else t * co[sl])
                        out[0, sl] += dx[a] * wy[b] * wz[c] * v
                        out[1, sl] += wx[a] * dy[b] * wz[c] * v
                        out[2, sl] += wx[a] * wy[b] * dz[c] * v
        return out

    def multiply_kphi(self, f):
        """In place: f times the inverse Laplacian, the deconvolution and 1/(mean density), DC = 0."""
        res, L = self.res, self.L
        kz, ky, kx = _wavenumbers(res, L, torch.float64)
        m, lap = res / L, self.c["lap"]

        def term(k):
            t = k / m
            return {0: lambda: -k * k, 2: lambda: -2 * (1 - torch.cos(t)) * m * m,
                    4: lambda: -(torch.cos(2 * t) - 16 * torch.cos(t) + 15) / 6 * m * m,
                    6: lambda: -(-2 * torch.cos(3 * t) + 27 * torch.cos(2 * t) - 270 * torch.cos(t) + 245) / 90
                    * m * m}[lap]()

        scale = res ** 3 / self.n ** 3 / self.c["resample"] ** 3
        mak = [torch.sinc(k / (2 * math.pi) / m) ** (-2 * self.W) if self.c["deconv"] else None for k in (kz, ky, kx)]
        tz, ty, tx = term(kz), term(ky), term(kx)
        for z in range(res):
            t = tz[z] + ty[0] + tx[0]
            if z == 0:
                t[0, 0] = 1.0
            v = scale / t
            if mak[0] is not None:
                v = v * (mak[0][z] * mak[1][0] * mak[2][0])
            if z == 0:
                v[0, 0] = 0.0
            f[z] *= v
        return f

    def potential(self, rho):
        res = self.res
        return torch.fft.irfftn(self.multiply_kphi(torch.fft.rfftn(rho)), s=(res, res, res))

    def difference(self, phi, axis, sign=-1.0):
        """sign times the central difference of the configured order along x, y or z (axis 0, 1, 2)."""
        h = self.L / self.res
        co = {2: (1 / 2,), 4: (8 / 12, -1 / 12), 6: (45 / 60, -9 / 60, 1 / 60)}[self.c["grad"]]
        dim = 2 - axis
        out = torch.zeros_like(phi)
        for j, c in enumerate(co, 1):
            out += (sign * c / h) * torch.roll(phi, -j, dim)
            out -= (sign * c / h) * torch.roll(phi, j, dim)
        return out

    def spawned(self, psi):
        """Positions of the resampled particle sets (Fourier interpolation of the sheet)."""
        n, L, nr = self.n, self.L, self.c["resample"]
        q = torch.arange(n, device=psi.device, dtype=torch.float64) * (L / n)
        m = torch.fft.fftfreq(n, device=psi.device, dtype=torch.float64)
        mh = torch.arange(n // 2 + 1, device=psi.device, dtype=torch.float64) / n
        for d in [(a / nr, b / nr, c / nr) for a in range(nr) for b in range(nr) for c in range(nr)][1:]:
            # the halved axis is z: the Nyquist phase is not Hermitian, so the choice of axis matters
            ph = torch.exp(2j * math.pi * (mh.view(-1, 1, 1) * d[2] + m.view(1, n, 1) * d[1] + m.view(1, 1, n) * d[0]))
            X = torch.empty((3, n, n, n), dtype=torch.float64, device=psi.device)
            for c, shape in enumerate(((1, 1, n), (1, n, 1), (n, 1, 1))):
                f = torch.fft.rfftn(psi[c].double(), dim=(1, 2, 0)) * ph
                X[c] = torch.fft.irfftn(f, s=(n, n, n), dim=(1, 2, 0)) + q.view(shape) + d[c] * L / n
            yield X.reshape(3, -1)

    def force(self, psi, W=None):
        W = W or self.W
        X = self.positions(psi)
        res = self.res
        acc = 0
        sets = list(self.spawned(psi)) if self.c["resample"] > 1 else []
        for s in self.shifts:
            rho = self.deposit(X, s, W)
            for Y in sets:
                rho += self.deposit(Y, s, W)
            if self.c["grad"] == 0:
                f = self.multiply_kphi(torch.fft.rfftn(rho))
                del rho
                for a, k in enumerate(reversed(_wavenumbers(res, self.L, torch.float64))):
                    kk = k.clone()
                    kk[kk.abs() > math.pi * res / self.L * (1 - 1e-9)] = 0.0
                    F = torch.fft.irfftn(-1j * kk * f, s=(res, res, res))
                    g = self.gather([F], X, s, W)
                    acc = acc + torch.nn.functional.pad(g, (0, 0, a, 2 - a))
                continue
            phi = self.potential(rho)
            del rho
            for a in range(3):
                F = self.difference(phi, a)
                acc = acc + torch.nn.functional.pad(self.gather([F], X, s, W), (0, 0, a, 2 - a))
                del F
        return (acc / len(self.shifts)).view(3, self.n, self.n, self.n)

    def fields(self, psi):
        """[delta, F_x, F_y, F_z] of the unshifted particles."""
        X = self.positions(psi)
        rho = self.deposit(X, (0, 0, 0), self.W)
        phi = self.potential(rho)
        return torch.stack([rho * (self.res ** 3 / self.n ** 3) - 1] + [self.difference(phi, a) for a in range(3)])

    def force_vjp(self, psi, abar):
        X = self.positions(psi)
        ab = abar.double().reshape(3, -1) / len(self.shifts)
        out = 0
        for s in self.shifts:
            phi = self.potential(self.deposit(X, s, self.W))
            G = [self.difference(phi, a) for a in range(3)]
            del phi
            out = out + self.gather_grad(G, list(ab), X, s, self.W)
            del G
            back = 0
            for a in range(3):
                back = back + self.difference(self.deposit(X, s, self.W, ab[a]), a, sign=1.0)
            # the inverse transform of the potential is real and symmetric: the same operator again
            out = out + self.gather_grad([self.potential(back)], [None], X, s, self.W)
        return out.view(3, self.n, self.n, self.n)


def _net64(params, case, x):
    """The network in float64: 27 shifted matrix products per layer; x (cin, r, r, r)."""
    off, r = 0, x.shape[1]
    taps = [(z, y, v) for z in (-1, 0, 1) for y in (-1, 0, 1) for v in (-1, 0, 1)]
    a = x.double()
    for l, (ci, co, cp, op) in enumerate(_net_layout(case)):
        w = params[off:off + 27 * cp * op].view(27, cp, op)
        b = params[off + 27 * cp * op:off + 27 * cp * op + op]
        off += 27 * cp * op + op
        y = b[:co].view(co, 1).expand(co, r ** 3)
        for t, (dz, dy, dx) in enumerate(taps):
            sh = torch.roll(a, (-dz, -dy, -dx), (1, 2, 3)).reshape(ci, -1)
            y = y + w[t, :ci, :co].t() @ sh
        a = (torch.relu(y) if l < NN_LAYERS - 1 else y).view(co, r, r, r)
    return a


def _exact_pk(case, psi):
    res, L, bins = case["res"], case["L"], PK_BINS
    pm = _PM64(dict(case, W=2))
    rho = pm.deposit(pm.positions(psi), (0, 0, 0), 2)
    p = torch.fft.rfftn(rho * (res ** 3 / case["n"] ** 3) - 1).abs() ** 2 * (L ** 3 / res ** 6)
    kz, ky, kx = _wavenumbers(res, L, torch.float64)
    k = torch.sqrt(kx * kx + ky * ky + kz * kz)
    lo, hi = math.log10(2 * math.pi / L), math.log10(math.pi * res / L * math.sqrt(3))
    edges = torch.tensor([10.0 ** ((1 - i / bins) * lo + i / bins * hi) for i in range(bins + 1)], device=DEV,
                         dtype=torch.float64)
    half = torch.ones(res // 2 + 1, device=DEV, dtype=torch.float64)
    half[0] = half[-1] = 0.5
    w = half.view(1, 1, -1).expand_as(k).reshape(-1)
    which = torch.bucketize(k.reshape(-1), edges, right=True) - 1
    ok = (which >= 0) & (which < bins)
    ids = which[ok]
    cnt = torch.bincount(ids, minlength=bins)
    ksum = torch.bincount(ids, weights=k.reshape(-1)[ok], minlength=bins)
    psum = torch.bincount(ids, weights=(p.reshape(-1) * w)[ok], minlength=bins)
    wsum = torch.bincount(ids, weights=w[ok], minlength=bins)
    empty = cnt == 0
    mid = torch.sqrt(edges[:-1] * edges[1:])
    kc = torch.where(empty, mid, ksum / cnt.clamp_min(1))
    return kc.cpu().numpy(), torch.where(empty, 0, psum / wsum.clamp_min(0.5)).cpu().numpy(), cnt.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("netforward", "netgrads", "corrected"):
        params = _net_params(case, seed).to(DEV).double()
    if kind == "netforward":
        return _net64(params, case, _net_meshes(case, seed)[0])
    if kind == "netgrads":
        x, t = _net_meshes(case, seed)
        params.requires_grad_(True)
        loss = torch.mean((_net64(params, case, x) - t.double()) ** 2)
        (g,) = torch.autograd.grad(loss, params)
        return float(loss), g.cpu().numpy()
    psi, mom = _displacements(case, seed)
    if kind == "pk":
        return _exact_pk(case, psi)
    pm = _PM64(case)
    if kind == "force":
        return pm.force(psi)
    if kind == "vjp":
        return pm.force_vjp(psi, _cotangents(case, seed)[0])
    coef = list(zip(*_coefficients(case)))
    if kind == "stepvjp":
        dd1, alpha, beta, dd2 = coef[0]
        pb, mb = (b.double() for b in _cotangents(case, seed))
        mb = mb + dd2 * pb
        pb = pb + pm.force_vjp(psi.double() + dd1 * mom.double(), beta * mb)
        return pb, alpha * mb + dd1 * pb
    p, m = psi.double(), mom.double()
    del psi, mom
    for dd1, alpha, beta, dd2 in coef:
        p = p + dd1 * m
        a = pm.force(p)
        if kind == "corrected":
            f = pm.fields(p)
            f[0] *= NN_SCALES["delta_scale"]
            f[1:] *= NN_SCALES["force_scale"]
            y = _net64(params, case, f)
            a = a + NN_SCALES["out_scale"] * pm.gather(list(y), pm.positions(p), (0, 0, 0), case["W"]).view_as(a)
        m = alpha * m + beta * a
        p = p + dd2 * m
    if kind == "hostrun":
        return p.permute(3, 2, 1, 0).cpu().numpy(), m.permute(3, 2, 1, 0).cpu().numpy()
    return p, m
