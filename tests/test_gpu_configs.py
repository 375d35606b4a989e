"""GPU parity at the benchmark configurations.

* 64³ particles / 128³ mesh, L = 250, 2LPT at a = 0.02, CIC, grad 2, BullFrog 10 steps
  to a = 1: the full run against the float64 oracle (positions, momenta, P(k)).
  The float32 floor of this run (float32 CPU port vs float64 oracle) is 8.8e-6 in Ψ,
  2.2e-5 in P, 8.4e-7 in max|ΔX|/L and 1.3e-6 in P(k).
* 256³ / 512³, L = 500, TSC, interlacing, order-4 gradient and Laplacian, FastPM
  (40-step schedule): the first two steps, and the whole 40-step run to a = 1, against
  the float64 C port (displacements, momenta, positions, P(k) per bin).
* 512³ / 1024³, L = 1000, 3LPT, PCS, interlacing, order-6 gradient, BullFrog (the
  throughput configuration): the first two steps against the float64 C port, which
  covers the 1024³-only paths (fused z pass, 16³ bricks in Morton order, box bounds).
* The reference's own physics check (test/nbody_parity_tests.jl:68-90): a
  fundamental plane wave grows as D(a) for every stepper, converging with resolution.
* 512³ / 1024³ (the throughput configuration), size-independent properties: the
  total PM force vanishes (momentum conservation of the symmetric scheme), repeated
  force calls agree, a step keeps the state finite.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

COSMO = dict(Omega_c=0.31 - 0.049, Omega_b=0.049, h=0.677, n_s=0.965, sigma8=0.81)


@pytest.fixture(scope="module")
def djb(cuda_device):
    import djb200
    return djb200


@pytest.fixture(scope="module")
def cosmo_pair(djb):
    from oracle import cosmology as cz
    return djb.Cosmology(**COSMO), cz.compute_timetables(cz.Cosmology(**COSMO))


def _ics(djb, cosmo, n, L, order, seed, device="cpu"):
    import torch

    from djb200 import ics
    dt = torch.float64 if device == "cpu" else torch.float32
    psi, pi = ics.lpt_ics(cosmo, n, L, 0.02, n_order=order, seed=seed, device=device, dtype=dt)
    return psi, pi


def test_c1_lcdm_bullfrog_vs_float64_oracle(djb, cosmo_pair):
    from oracle import nbody as onb
    from oracle import pm as opm
    from oracle import power as opw
    cl, co = cosmo_pair
    n, res, L = 64, 128, 250.0
    psi, pi = _ics(djb, cl, n, L, 2, seed=7)
    psi, pi = psi.numpy(), pi.numpy()
    kw = dict(boxsize=L, a_ini=0.02, a_end=1.0, n_steps=10, res_pm=res, stepper="bullfrog", worder=2,
              grad_kernel_order=2, antialias=0)
    P64, M64, _ = onb.run_nbody(co, psi, pi, return_displacement=True, **kw)
    Pg, Mg, _ = djb.run_nbody(cl, psi.astype(np.float32), pi.astype(np.float32), return_displacement=True, **kw)
    assert rel(Pg, P64) < 2e-5
    assert np.max(np.abs(Pg - P64)) / L < 1e-5        # positions, relative to the box
    assert rel(Mg, M64) < 5e-5
    # P(k) of the final particles, 32 log bins: GPU (CIC deposit + float64 shells) vs oracle
    cfg = djb.PMConfig(res_pm=res, n_part=n, boxsize=L, worder=2, grad_order=2)
    with djb.PMSolver(cfg) as S:
        S.set_state(Pg, Mg)
        k, pk, nm = S.state_power_spectrum(bins=32)
    X = onb.add_q(P64, L).reshape(-1, 3)
    mesh = opm.pm_scatter(np.zeros((res, res, res)), X, res, L, 2)
    kr, pkr, nmr = opw.evaluate_power_spectrum(opw.density_contrast(mesh, n), L, bins=32)
    assert np.array_equal(nm, nmr)
    nz = nmr > 0
    assert np.max(np.abs(pk[nz] / pkr[nz] - 1)) < 1e-4


def test_c2_tsc_interlaced_fastpm_first_steps_vs_float64(djb, cosmo_pair):
    from oracle import cpm
    from oracle import pm as opm
    cl, co = cosmo_pair
    n, res, L = 256, 512, 500.0
    psi_t, pi_t = _ics(djb, cl, n, L, 2, seed=11, device="cuda")
    psi, pi = psi_t.cpu().numpy().astype(np.float64), pi_t.cpu().numpy().astype(np.float64)
    del psi_t, pi_t
    coef = djb.stepper_coefficients(cl, "fastpm", 0.02, 1.0, 40)
    cfg = djb.PMConfig(res_pm=res, n_part=n, boxsize=L, worder=3, antialias=1, grad_order=4, lap_order=4)
    with djb.PMSolver(cfg) as S:
        S.set_state(psi.astype(np.float32), pi.astype(np.float32))
        for k in range(2):
            S.step(coef["ddrift1"][k], coef["alpha"][k], coef["beta"][k], coef["ddrift2"][k])
        Pg, Mg = S.get_state()
    C = cpm.CPUPM(opm.PMConfig(res_pm=res, n_part=n, boxsize=L, worder=3, antialias=1, grad_order=4,
                               lap_order=4), dtype=np.float64)
    p64, m64 = psi.astype(np.float32).astype(np.float64), pi.astype(np.float32).astype(np.float64)
    for k in range(2):
        p64, m64 = C.step(p64, m64, coef["ddrift1"][k], coef["alpha"][k], coef["beta"][k], coef["ddrift2"][k])
    assert rel(Pg, p64) < 2e-5
    assert rel(Mg, m64) < 5e-5


def _report(capsys, name, **errs):
    with capsys.disabled():
        print(f"\n[{name}] " + ", ".join(f"{k} = {v:.3e}" for k, v in errs.items()))


def _port_run(C, p64, m64, coef, k0, k1):
    for k in range(k0, k1):
        p64, m64 = C.step(p64, m64, coef["ddrift1"][k], coef["alpha"][k], coef["beta"][k], coef["ddrift2"][k])
    return p64, m64


@pytest.mark.slow
def test_c2_full_fastpm_run_vs_float64(djb, cosmo_pair, capsys):
    """The whole 40-step FastPM run of 256³ particles on a 512³ mesh (TSC, interlacing,
    order-4 gradient and Laplacian) from a = 0.02 to 1, float32 on the GPU against the
    float64 C port from the same float32 ICs. Bars: positions max|ΔX|/L < 1e-5 (the
    target's relative 1e-5 in positions); P(k) of the final particles per bin < 1e-4;
    displacements and momenta, which carry float32 round-off amplified by 40 steps of
    gravitational growth, < 2e-4 and 5e-4 of their largest entries."""
    from oracle import cpm
    from oracle import nbody as onb
    from oracle import pm as opm
    from oracle import power as opw
    cl, co = cosmo_pair
    n, res, L = 256, 512, 500.0
    psi_t, pi_t = _ics(djb, cl, n, L, 2, seed=11, device="cuda")
    psi = psi_t.cpu().numpy().astype(np.float32)
    pi = pi_t.cpu().numpy().astype(np.float32)
    del psi_t, pi_t
    coef = djb.stepper_coefficients(cl, "fastpm", 0.02, 1.0, 40)
    opts = dict(worder=3, antialias=1, grad_order=4, lap_order=4)
    with djb.PMSolver(djb.PMConfig(res_pm=res, n_part=n, boxsize=L, **opts)) as S:
        S.set_state(psi, pi)
        S.run(coef["ddrift1"], coef["alpha"], coef["beta"], coef["ddrift2"])
        Pg, Mg = S.get_state()
        k, pk, nm = S.state_power_spectrum(bins=32)
    C = cpm.CPUPM(opm.PMConfig(res_pm=res, n_part=n, boxsize=L, **opts), dtype=np.float64)
    p64, m64 = _port_run(C, psi.astype(np.float64), pi.astype(np.float64), coef, 0, 40)
    # P(k) of the float64 final state: CIC deposit (the C port), δ, float64 shell sums
    X = onb.add_q(p64, L)
    mesh = np.zeros(res ** 3)
    Xb = np.ascontiguousarray(np.moveaxis(X, -1, 0).transpose(0, 3, 2, 1))  # [c][k][j][i]
    cpm.lib().cpm_scatter_f64(cpm._ptr(Xb), n ** 3, res, float(L), 2, cpm._ptr(mesh))
    field = mesh.reshape(res, res, res).T                                    # [ix,iy,iz]
    kr, pkr, nmr = opw.evaluate_power_spectrum(opw.density_contrast(field, n), L, bins=32)
    dx = np.abs(Pg.astype(np.float64) - p64)
    errs = dict(psi=rel(Pg, p64), mom=rel(Mg, m64), dX_over_L=float(dx.max()) / L,
                pk=float(np.max(np.abs(pk[nmr > 0] / pkr[nmr > 0] - 1))))
    _report(capsys, "C2 40-step FastPM vs float64", **errs)
    # measured on the B200: psi 6.0e-5, mom 2.0e-4, dX/L 4.2e-6, P(k) 2.0e-6
    assert np.array_equal(nm, nmr)
    assert errs["dX_over_L"] < 1e-5
    assert errs["pk"] < 1e-4
    assert errs["psi"] < 2e-4 and errs["mom"] < 5e-4


@pytest.mark.slow
def test_c3_bullfrog_steps_vs_float64_port(djb, cosmo_pair, capsys):
    """512³ particles on the 1024³ mesh, L = 1000, 3LPT ICs at a = 0.02, PCS,
    interlacing, order-6 gradient, BullFrog (20-step schedule): the first two steps,
    float32 on the GPU against the float64 C port from the same float32 ICs. The
    momentum after the first step isolates one force evaluation (Mom₁ = α Mom₀ + β F)."""
    import psutil

    from oracle import cpm
    from oracle import pm as opm
    if psutil.virtual_memory().available < 160 * 2 ** 30:
        pytest.skip("the float64 port at 1024³ needs about 80 GB of host memory (160 GB free asked)")
    cl, co = cosmo_pair
    n, res, L = 512, 1024, 1000.0
    psi_t, pi_t = _ics(djb, cl, n, L, 3, seed=5, device="cuda")
    psi = psi_t.cpu().numpy().astype(np.float32)
    pi = pi_t.cpu().numpy().astype(np.float32)
    del psi_t, pi_t
    coef = djb.stepper_coefficients(cl, "bullfrog", 0.02, 1.0, 20)
    opts = dict(worder=4, antialias=1, grad_order=6)
    got = []
    with djb.PMSolver(djb.PMConfig(res_pm=res, n_part=n, boxsize=L, **opts)) as S:
        S.set_state(psi, pi)
        for k in range(2):
            S.step(coef["ddrift1"][k], coef["alpha"][k], coef["beta"][k], coef["ddrift2"][k])
            got.append(S.get_state())
    C = cpm.CPUPM(opm.PMConfig(res_pm=res, n_part=n, boxsize=L, **opts), dtype=np.float64)
    p64, m64 = psi.astype(np.float64), pi.astype(np.float64)
    del psi, pi
    errs = {}
    for k in range(2):
        p64, m64 = _port_run(C, p64, m64, coef, k, k + 1)
        Pg, Mg = got[k]
        errs[f"psi{k + 1}"] = rel(Pg, p64)
        errs[f"mom{k + 1}"] = rel(Mg, m64)
        errs[f"dX{k + 1}_over_L"] = float(np.max(np.abs(Pg.astype(np.float64) - p64))) / L
    _report(capsys, "C3 BullFrog steps vs float64", **errs)
    # measured on the B200: psi 9.3e-6 / 1.5e-5, mom 2.8e-5 / 2.1e-5, dX/L 2.1e-8 / 5.6e-8;
    # the momentum bar is the one of the other configurations (float32 transforms of 1024³)
    for k in (1, 2):
        assert errs[f"psi{k}"] < 2e-5
        assert errs[f"mom{k}"] < 5e-5
        assert errs[f"dX{k}_over_L"] < 1e-5


@pytest.mark.parametrize("stepper,nsteps", [("bullfrog", 1), ("bullfrog", 16), ("fastpm", 16), ("symplectic", 64)])
def test_plane_wave_linear_growth(djb, stepper, nsteps):
    """nbody_parity_tests.jl:68-90: growth error < 1e-2 at 32³ and converging (16³→32³ > 3x)."""
    c = djb.Cosmology("Planck18EEBAOSN")
    L, a0 = 100.0, 0.05
    D0, D1 = c.Dplus(a0), c.Dplus(1.0)
    err = {}
    for n in (16, 32):
        q = np.array([i * L / n for i in range(n)])
        psi1 = np.zeros((n, n, n, 3))
        psi1[..., 0] = (1e-3 * np.sin(2 * np.pi * q / L))[:, None, None]
        Psi, _, _ = djb.run_nbody(c, (D0 * psi1).astype(np.float32), psi1.astype(np.float32), boxsize=L, a_ini=a0,
                                  a_end=1.0, n_steps=nsteps, res_pm=2 * n, stepper=stepper, return_displacement=True)
        Psi = Psi.astype(np.float64)
        # stays one-dimensional up to float32 round-off: positions X = q + Ψ near q ≈ L carry
        # an ulp of 7.6e-6, 0.8% of the 1e-3 wave, and the transverse leak stays ~2e-5 of
        # the wave (the reference's 1e-12 bar is for Float64)
        assert np.max(np.abs(Psi[..., 1:])) < 1e-4 * np.max(np.abs(Psi[..., 0]))
        err[n] = abs(np.sum(Psi[..., 0] * psi1[..., 0]) / np.sum(psi1[..., 0] ** 2) / D1 - 1)
    assert err[32] < 1e-2
    assert err[16] / err[32] > 3


@pytest.mark.slow
def test_c3_throughput_config_properties(djb):
    """512³ / 1024³, PCS, interlacing, grad 6: the sum of all PM forces vanishes, two
    force calls agree, and a BullFrog step keeps the state finite."""
    import torch
    c = djb.Cosmology(**COSMO)
    n, res, L = 512, 1024, 1000.0
    psi, pi = _ics(djb, c, n, L, 3, seed=5, device="cuda")
    cfg = djb.PMConfig(res_pm=res, n_part=n, boxsize=L, worder=4, antialias=1, grad_order=6)
    psi_d = djb.native_view(psi.float())
    pi_d = djb.native_view(pi.float())
    del psi, pi
    with djb.PMSolver(cfg) as S:
        a1 = S.acceleration(psi_d)
        a2 = S.acceleration(psi_d)
        tot = a1.double().sum(dim=(1, 2, 3))
        scale = a1.double().abs().sum(dim=(1, 2, 3))
        assert float((tot.abs() / scale).max()) < 1e-5          # momentum conservation
        assert float((a1 - a2).abs().max() / a1.abs().max()) < 1e-5  # float atomics reorder only
        co = djb.stepper_coefficients(c, "bullfrog", 0.02, 1.0, 20)
        S.set_state(psi_d, pi_d)
        S.step(co["ddrift1"][0], co["alpha"][0], co["beta"][0], co["ddrift2"][0])
        p, m = S.get_state(device=True)
        assert bool(torch.isfinite(p).all()) and bool(torch.isfinite(m).all())
        assert float((p - psi_d).abs().max()) > 0


def test_fused_z_pass_matches_3d_transforms(djb, monkeypatch):
    """1024^3 mesh: the batched 2-D transforms with the fused z pass (forward z DFT, Kφ,
    inverse z DFT in one kernel) against the 3-D cuFFT transforms with the separate
    k-space multiplication (DJB_ZPASS=0), on strongly clustered particles."""
    n, res, L = 64, 1024, 1000.0
    rng = np.random.default_rng(3)
    psi = (20 * rng.standard_normal((n, n, n, 3))).astype(np.float32)
    cfg = djb.PMConfig(res_pm=res, n_part=n, boxsize=L, worder=4, antialias=1, grad_order=6, deconvolve=True)
    with djb.PMSolver(cfg) as A:
        a = A.acceleration(psi)
    monkeypatch.setenv("DJB_ZPASS", "0")
    with djb.PMSolver(cfg) as B:
        b = B.acceleration(psi)
    assert rel(a, b) < 1e-5


@pytest.mark.parametrize("res,n,W,lap,dec", [(128, 50, 4, 0, True), (256, 64, 3, 4, False), (512, 48, 2, 0, False),
                                             (512, 70, 4, 6, True)])
def test_fused_z_pass_sizes_match_3d_transforms(djb, monkeypatch, res, n, W, lap, dec):
    """The fused z pass at its smaller sizes (one kernel instance each; rows of res/2 + 1 pencils,
    so most tiles of 16 consecutive pencils straddle two ky) against the 3-D transforms with
    the separate multiplication. Both
    are float32 transforms of the same density: a few 1e-7 per transform, amplified by the
    deconvolution; 1e-5 as at 1024^3."""
    rng = np.random.default_rng(res + n)
    L = 100.0
    psi = (5 * rng.standard_normal((n, n, n, 3))).astype(np.float32)
    cfg = djb.PMConfig(res_pm=res, n_part=n, boxsize=L, worder=W, antialias=1, grad_order=4, lap_order=lap,
                       deconvolve=dec)
    with djb.PMSolver(cfg) as A:
        a = A.acceleration(psi)
    monkeypatch.setenv("DJB_ZPASS", "0")
    with djb.PMSolver(cfg) as B:
        b = B.acceleration(psi)
    assert rel(a, b) < 1e-5


def _multiplier64(cfg, ky):
    """The multiplier on the modes [kz][kx] of one ky in float64, and 0 at the zero mode."""
    res, L = cfg.res_pm, cfg.boxsize
    m = res / L
    i = np.arange(res)
    k = np.where(i < res // 2, i, i - res) * 2 * np.pi / L
    t = k / m
    T = {0: -k * k, 2: -2 * (1 - np.cos(t)) * m * m,
         4: -(np.cos(2 * t) - 16 * np.cos(t) + 15) / 6 * (m * m),
         6: -(-2 * np.cos(3 * t) + 27 * np.cos(2 * t) - 270 * np.cos(t) + 245) / 90 * (m * m)}[cfg.lap_order]
    M = np.sinc(t / (2 * np.pi)) ** (-2.0 * cfg.worder) if cfg.deconvolve else np.ones(res)
    nh = res // 2 + 1
    s0 = 1.0 / cfg.n_part ** 3
    with np.errstate(divide="ignore"):
        K = s0 / ((T[:nh] + T[ky])[None, :] + T[:, None]) * (M[:nh] * M[ky])[None, :] * M[:, None]
    if ky == 0:
        K[0, 0] = 0.0
    return K


@pytest.mark.parametrize("res,L", [(128, 100.0), (256, 3.0e-9), (512, 1000.0), (1024, 2.0e6)])
def test_fused_multiplier_is_the_float64_quotient(djb, res, L):
    """The fused z pass' multiplier against float64, mode by mode, for every Laplacian with and
    without deconvolution and in any unit of length: rounded once, so half a unit in the last
    place (and 1e-3 of one for the float64 cosines of the finite-difference terms, whose
    cancellation near k = 0 costs up to 1e5 of their 1e-16). The general passes are compared
    with the same bound; the two differ only where the quotient lies that close to a tie."""
    import ctypes as C

    from djb200 import _lib
    got = [np.empty((res, res // 2 + 1), dtype=np.float32) for _ in range(2)]
    step = max(1, res // 64)
    for lap in (0, 2, 4, 6):
        for dec in (False, True):
            cfg = djb.PMConfig(res_pm=res, n_part=16, boxsize=L, worder=4, grad_order=4, lap_order=lap,
                               deconvolve=dec)
            with djb.PMSolver(cfg) as S:
                differ = 0
                for ky in sorted({0, 1, res // 2 - 1, res // 2, res - 1, *range(0, res, step)}):
                    ref = _multiplier64(cfg, ky)
                    ulp = np.spacing(np.abs(ref).astype(np.float32)).astype(np.float64)
                    for fused in (0, 1):
                        _lib.check(_lib.lib.djb_selftest_multiplier(S.handle, ky, fused,
                                                                    C.c_void_p(got[fused].ctypes.data)))
                        assert np.max(np.abs(got[fused] - ref) / ulp) <= 0.5 + 1e-3, (lap, dec, ky, fused)
                    differ += int(np.sum(got[0] != got[1]))
                assert differ <= 2, (lap, dec)
