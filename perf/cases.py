"""Performance cases: the work that programs built on this library have it do.

Every case goes through the public entry points (the Python handles over the C
ABI, or the C ABI itself where the library's own training loop calls it) and
covers one of these uses:

  cells   N independent cells stepped with the Cell interface's update()
  strand  one recorded 1D strand run to its stop time (the OneD driver)
  sweep   a batch of uneven single cells and strands in one launch
  sheet   a 2D sheet stepped by the tissue simulation
  shell   a 3D ventricular shell with rotating fibres stepped by the tissue
          simulation
  train   mini-batches of the surrogate's training (normalise, forward,
          backward, Adam)
  infer   the surrogate's network on a block of rows

Tissue and cell states are taken from one paced beat of the cell model, so that
a pass sees rest, upstroke, plateau and repolarisation side by side, as a wave
that has crossed part of the tissue leaves them.  The beat, the geometries and
the 64-bit results (`exact`) are computed here with numpy and torch alone.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import lqt1_gb300 as lq
from lqt1_gb300 import _native, surrogate

DT = 0.02                      # ms, the step of every reference driver
ENDO, MID, EPI, EMPTY = 3, 4, 2, 255
D_FIBRE, D_TRANS = 0.154, 0.0385     # mm^2/ms
WARM = 100                     # steps a tissue simulation has taken before the pass (2 ms)
RING = 32                      # pinned buffers of a per-step read-back

# scenario factors: GKs, PCa, GKs under ISO, ISO shifts of the d and f gates
MODELS = {
    "cpu": ("default", {}, (1.0, 1.6, 3.2, 12.0, 8.0)),
    "shell": ("baseline", dict(gks_scale=0.5, pca_scale=2.0, gks_iso_scale=1.5), (0.5, 2.0, 1.5, 0.0, 0.0)),
    "sheet": ("lqt1", dict(gks_scale=0.5), (0.5, 1.0, 1.0, 0.0, 0.0)),
}


# ---- the cases -------------------------------------------------------------------
def listed():
    return [
        # the SingleCell loop: one cell, one update, V read after it
        dict(name="cell_one_update", kind="cells", n=1, steps=1, fp64=False),
        # a population of cells over 20 ms of an action potential
        dict(name="cells_population", kind="cells", n=20011, steps=1000, fp64=False),
        # the OneD driver's strand (100 cells), V and pseudo-ECG every 10 steps
        dict(name="strand_recorded", kind="strand", n=100, ms=20.0, fp64=False),
        # parameter sweep: single cells and strands of 50..400 cells, uneven ends
        dict(name="sweep_uneven", kind="sweep", instances=1024, ms=30.0),
        # a small sheet at the start of a beat: S1, activation, detectors, whole state
        dict(name="sheet_small_s1", kind="sheet", nx=97, ny=64, steps=100, fp64=False, sur=False, fibre=True,
             readback=False, phase=-20.0, s1=True),
        # the S1-S2 sheet workload's size, wave half across
        dict(name="sheet_600", kind="sheet", nx=600, ny=600, steps=50, fp64=False, sur=False, fibre=False,
             readback=False, phase=60.0, s1=False),
        # surrogate steps with V of every voxel read back after every step
        dict(name="sheet_sur_readback", kind="sheet", nx=200, ny=200, steps=20, fp64=False, sur=True, fibre=False,
             readback=True, phase=150.0, s1=False),
        # the FP64 form on a small shell
        dict(name="shell_fp64", kind="shell", nx=70, nz=90, steps=10, fp64=True, sur=False, ecg=False, phase=30.0),
        # the mixed form on the accuracy shell's grid (170 x 170 x 220)
        dict(name="shell_mixed", kind="shell", nx=170, nz=220, steps=50, fp64=False, sur=False, ecg=False,
             phase=40.0),
        # the headline: whole ventricle, surrogate macro steps, six electrodes
        dict(name="ventricle_surrogate", kind="shell", nx=320, nz=420, steps=50, fp64=False, sur=True, ecg=True,
             phase=120.0),
        # surrogate training: 16 mini-batches of the recipe's size
        dict(name="train_batches", kind="train", batch=8192, steps=16),
        # surrogate inference on a validation block
        dict(name="infer_block", kind="infer", rows=1000003),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cells", "strand", "sweep", "sheet", "shell", "train", "infer"])
    if kind == "cells":
        fp64 = rng.random() < 0.3
        n = _log(rng, 1, 2000 if fp64 else 30000)
        return dict(kind=kind, n=n, steps=_log(rng, 1, 20 if fp64 else 1000), fp64=fp64)
    if kind == "strand":
        fp64 = rng.random() < 0.2
        return dict(kind=kind, n=_log(rng, 20, 500), ms=round(rng.uniform(0.5, 2.0) * (1 if fp64 else 10), 2),
                    fp64=fp64)
    if kind == "sweep":
        return dict(kind=kind, instances=_log(rng, 30, 1000), ms=round(rng.uniform(8.0, 30.0), 2))
    if kind == "sheet":
        sur = rng.random() < 0.4
        fp64 = not sur and rng.random() < 0.2
        top = 100 if fp64 else 600
        return dict(kind=kind, nx=_log(rng, 24, top), ny=_log(rng, 24, top),
                    steps=10 if fp64 else rng.choice([20, 50, 100]), fp64=fp64, sur=sur, fibre=rng.random() < 0.5,
                    readback=rng.random() < 0.3, phase=round(rng.uniform(5.0, 400.0), 1), s1=rng.random() < 0.3)
    if kind == "shell":
        sur = rng.random() < 0.5
        fp64 = not sur and rng.random() < 0.3
        nx = _log(rng, 48, 70 if fp64 else 200)
        return dict(kind=kind, nx=nx, nz=int(nx * rng.uniform(1.2, 1.4)),
                    steps=10 if fp64 else rng.choice([20, 50, 100]), fp64=fp64, sur=sur, ecg=rng.random() < 0.5,
                    phase=round(rng.uniform(5.0, 400.0), 1))
    if kind == "train":
        return dict(kind=kind, batch=16 * _log(rng, 16, 512), steps=rng.choice([4, 8, 16]))
    return dict(kind=kind, rows=_log(rng, 1000, 1000000))


# ---- the cell model in 64 bits (numpy or torch arrays) ------------------------------
def _tpord(xp, s, ct, par, dt, ist, dvgap):
    """One update of the TPORd cell (SingleCell/TPORd.cc:379-1021).  s: the 40
    states, each an array; ct: cell types; par: MODELS factors.  Returns the new
    states, the ionic dV/dt and (INa, ICaL, IKr, IKs, IK1)."""
    gks_f, pca_f, iso_f, dshift, fshift = par
    exp, log, where = xp.exp, xp.log, xp.where
    (v, nai, nass, ki, kss, cai, cass, cansr, cajsr, m, h, j, hsp, jp, mL, hL, hLp, a, iF, iS, ap, iFp, iSp, d, ff, fs,
     fcaf, fcas, jca, nca, ffp, fcafp, xrf, xrs, xs1, xs2, xk1, Jnp, Jp, CaMKt) = s
    epi, mid = ct == EPI, ct == MID

    one = 0.0 * v + 1.0

    def cls(endo, e, mm):
        return where(epi, e * one, where(mid, mm * one, endo * one))

    def sg(x):
        return 1.0 / (1.0 + exp(x))

    def relax(x, inf, rate):
        return inf - (inf - x) * exp(-dt * rate * one)

    nao, cao, ko, R, T, F = 140.0, 1.8, 5.4, 8314.0, 310.0, 96485.0
    L, rad = 0.01, 0.0011
    vcell = 1000 * 3.14 * rad * rad * L
    acap = 2 * (2 * 3.14 * rad * rad + 2 * 3.14 * rad * L)
    vmyo, vnsr, vjsr, vss = 0.68 * vcell, 0.0552 * vcell, 0.0048 * vcell, 0.02 * vcell
    ENa, EK = R * T / F * log(nao / nai), R * T / F * log(ko / ki)
    EKs = R * T / F * log((ko + 0.01833 * nao) / (ki + 0.01833 * nai))
    CaMKb = 0.05 * (1 - CaMKt) / (1 + 0.0015 / cass)
    fP = 1 / (1 + 0.15 / (CaMKb + CaMKt))
    vf, vff = v * F / (R * T), v * F * F / (R * T)
    # fast Na
    am = sg((-60 - v) / 5)
    bm = 0.1 * sg((v + 35) / 5) + 0.1 * sg((v - 50) / 200)
    minf = sg((-56.86 - v) / 9.03) ** 2
    up = v >= -40
    vlo = where(up, 0.0 * v - 40, v)
    vhi = where(up, v, 0.0 * v - 40)
    rh = where(up, 0.77 / (0.13 * (1 + exp(-(vhi + 10.66) / 11.1))),
               0.057 * exp(-(vlo + 80) / 6.8) + 2.7 * exp(0.079 * vlo) + 3.1e5 * exp(0.3485 * vlo))
    rj = where(up, 0.6 * exp(0.057 * vhi) / (1 + exp(-0.1 * (vhi + 32))),
               (-2.5428e4 * exp(0.2444 * vlo) - 6.948e-6 * exp(-0.04391 * vlo)) * (vlo + 37.78) /
               (1 + exp(0.311 * (vlo + 79.23))) + 0.02424 * exp(-0.01052 * vlo) / (1 + exp(-0.1378 * (vlo + 40.14))))
    hinf = sg((v + 71.55) / 7.43) ** 2
    m, h, j = relax(m, minf, 1 / (am * bm)), relax(h, hinf, rh), relax(j, hinf, rj)
    INa = 14.838 * m ** 3 * h * j * (v - ENa)
    # late Na
    mL = relax(mL, sg(-(v + 42.85) / 5.264), 6.765 * exp((v + 11.64) / 34.77) + 8.552 * exp(-(v + 77.42) / 5.955))
    hL, hLp = relax(hL, sg((v + 87.61) / 7.488), 1 / 200.), relax(hLp, sg((v + 93.81) / 7.488), 1 / 600.)
    INaL = cls(0.0075, 0.0045, 0.0075) * (v - ENa) * mL * ((1 - fP) * hL + fP * hLp)
    # transient outward
    ta = 1.0515 / (sg(-(v - 18.4099) / 29.3814) / 1.2089 + 3.5 * sg((v + 100) / 29.3814))
    iss = sg((v + 43.94) / 5.711)
    delta = where(epi, 1 - 0.95 * sg((v + 70) / 5), one)
    tF = (4.562 + 1 / (0.3933 * exp(-(v + 100) / 100) + 0.08004 * exp((v + 50) / 16.59))) * delta
    tS = (23.62 + 1 / (0.001416 * exp(-(v + 96.52) / 59.05) + 1.780e-8 * exp((v + 114.1) / 8.079))) * delta
    AiF = sg((v - 213.6) / 151.2)
    dp = (1.354 + 1e-4 / (exp((v - 167.4) / 15.89) + exp(-(v - 12.23) / 0.2154))) * (1 - 0.5 * sg((v + 70) / 20))
    a, ap = relax(a, sg(-(v - 14.34) / 14.82), 1 / ta), relax(ap, sg(-(v - 24.34) / 14.82), 1 / ta)
    iF, iS = relax(iF, iss, 1 / tF), relax(iS, iss, 1 / tS)
    iFp, iSp = relax(iFp, iss, 1 / (dp * tF)), relax(iSp, iss, 1 / (dp * tS))
    Ito = cls(0.02, 0.08, 0.08) * (v - EK) * ((1 - fP) * a * (AiF * iF + (1 - AiF) * iS) +
                                             fP * ap * (AiF * iFp + (1 - AiF) * iSp))
    # L-type Ca
    td = 0.6 + 1 / (exp(-0.05 * (v + 6)) + exp(0.09 * (v + 14)))
    finf = sg((v + 19.58 + fshift) / 3.696)
    tff = 7 + 1 / (0.0045 * exp(-(v + 20) / 10) + 0.0045 * exp((v + 20) / 10))
    tfs = 1000 + 1 / (0.000035 * exp(-(v + 5) / 4) + 0.000035 * exp((v + 5) / 6))
    tcf = 7 + 1 / (0.04 * exp(-(v - 4) / 7) + 0.04 * exp((v - 4) / 7))
    tcs = 100 + 1 / (0.00012 * exp(-v / 3) + 0.00012 * exp(v / 7))
    Af = 0.3 + 0.6 * sg((v - 10) / 10)
    d = relax(d, sg(-(v + 3.94 + dshift) / 4.23), 1 / td)
    ff, fs, ffp = relax(ff, finf, 1 / tff), relax(fs, finf, 1 / tfs), relax(ffp, finf, 1 / (2.5 * tff))
    fcaf, fcas, fcafp = relax(fcaf, finf, 1 / tcf), relax(fcas, finf, 1 / tcs), relax(fcafp, finf, 1 / (2.5 * tcf))
    jca = relax(jca, finf, 1 / 75.)
    anca = 1 / (1000 / jca + (1 + 0.002 / cass) ** 4)
    nca = relax(nca, anca * 1000 / jca, jca)
    e1, e2 = exp(vf), exp(2 * vf)
    PCa = 0.0001 * pca_f * cls(1.0, 1.2, 2.5)
    gate = (1 - fP) * d * ((0.6 * ff + 0.4 * fs) * (1 - nca) + jca * (Af * fcaf + (1 - Af) * fcas) * nca) + \
        1.1 * fP * d * ((0.6 * ffp + 0.4 * fs) * (1 - nca) + jca * (Af * fcafp + (1 - Af) * fcas) * nca)
    ICaL = PCa * gate * 4 * vff * (cass * e2 - 0.341 * cao) / (e2 - 1)
    ICaNa = 0.00125 * PCa * gate * vff * 0.75 * (nass * e1 - nao) / (e1 - 1)
    ICaK = 3.574e-4 * PCa * gate * vff * 0.75 * (kss * e1 - ko) / (e1 - 1)
    # K currents
    xrinf = sg(-(v + 8.337) / 6.789)
    txf = 12.98 + 1 / (0.3652 * exp((v - 31.66) / 3.869) + 4.123e-5 * exp(-(v - 47.78) / 20.38))
    txs = 1.865 + 1 / (0.06629 * exp((v - 34.70) / 7.355) + 1.128e-5 * exp(-(v - 29.74) / 25.94))
    Axf = sg((v + 54.81) / 38.21)
    xrf, xrs = relax(xrf, xrinf, 1 / txf), relax(xrs, xrinf, 1 / txs)
    IKr = 0.046 * cls(1.0, 1.3, 0.8) * (Axf * xrf + (1 - Axf) * xrs) * sg((v + 55) / 75) * sg((v - 10) / 30) * (v - EK)
    xsinf = sg(-(v + 11.6) / 8.932)
    t1 = 817.3 + 1 / (2.326e-4 * exp((v + 48.28) / 17.8) + 0.001292 * exp(-(v + 210) / 230))
    xs1 = relax(xs1, xsinf, 1 / t1)
    xs2 = relax(xs2, xsinf, 0.01 * exp((v - 50) / 20) + 0.0193 * exp(-(v + 66.54) / 31))
    GKs = 0.0034 * gks_f * iso_f * cls(1.0, 1.4, 1.0)
    IKs = GKs * (1 + 0.6 / (1 + (3.8e-5 / cai) ** 1.4)) * xs1 * xs2 * (v - EKs)
    xkinf = sg(-(v + 2.5538 * ko + 144.59) / (1.5692 * ko + 3.8115))
    xk1 = relax(xk1, xkinf, (exp(-(v + 127.2) / 20.36) + exp((v + 236.8) / 69.33)) / 122.2)
    IK1 = 0.1908 * cls(1.0, 1.2, 1.3) * math.sqrt(ko) * sg((v + 105.8 - 2.6 * ko) / 9.493) * xk1 * (v - EK)
    # Na/Ca exchange
    kna1, kna2, kna3, kas = 15.0, 5.0, 88.12, 12.5
    hca, hna = exp(0.167 * vf), exp(0.5224 * vf)
    h7 = 1 + nao / kna3 * (1 + 1 / hna)
    h8, h9 = nao / (kna3 * hna * h7), 1 / h7
    h10 = kas + 1 + nao / kna1 * (1 + nao / kna2)
    k1, k2, k5 = 1 / h10 * cao * 1.5e6, 5e3, 5e3
    k3p, k3pp = h9 * 6e4, h8 * 5e3
    k3, k8 = k3p + k3pp, h8 * nao * nao / (h10 * kna1 * kna2) * 6e4

    def exchange(na, ca):
        h1 = 1 + na / kna3 * (1 + hna)
        h2, h3 = na * hna / (kna3 * h1), 1 / h1
        h4 = 1 + na / kna1 * (1 + na / kna2)
        h5, h6 = na * na / (h4 * kna1 * kna2), 1 / h4
        k4p, k4pp = h3 * 6e4 / hca, h2 * 5e3
        k4, k6, k7 = k4p + k4pp, h6 * ca * 1.5e6, h5 * h2 * 6e4
        x1 = k2 * k4 * (k7 + k6) + k5 * k7 * (k2 + k3)
        x2 = k1 * k7 * (k4 + k5) + k4 * k6 * (k1 + k8)
        x3 = k1 * k3 * (k7 + k6) + k8 * k6 * (k2 + k3)
        x4 = k2 * k8 * (k4 + k5) + k3 * k5 * (k1 + k8)
        t = x1 + x2 + x3 + x4
        E1, E2, E3, E4 = x1 / t, x2 / t, x3 / t, x4 / t
        jna = 3 * (E4 * k7 - E1 * k8) + E3 * k4pp - E2 * k3pp
        return 0.0008 * cls(1.0, 1.1, 1.4) / (1 + (150e-6 / ca) ** 2) * (jna + 2 * (E2 * k2 - E1 * k1))

    Ii, Iss = 0.8 * exchange(nai, cai), 0.2 * exchange(nass, cass)
    # Na/K pump
    Knai, Knao = 9.073 * exp(-0.155 * vf / 3), 27.78 * exp(1.155 * vf / 3)
    P = 4.2 / (1 + 1e-7 / 1.698e-7 + nai / 224.0 + ki / 292.0)
    rn, ro, rk, rko = nai / Knai, nao / Knao, ki / 0.5, ko / 0.3582
    di, do = (1 + rn) ** 3 + (1 + rk) ** 2 - 1, (1 + ro) ** 3 + (1 + rko) ** 2 - 1
    atp = 9.8 / 1.698e-7
    a1, b1, a2, b2 = 949.5 * rn ** 3 / di, 182.4 * 0.05, 687.2, 39.4 * ro ** 3 / do
    a3, b3 = 1899.0 * rko ** 2 / do, 79300.0 * P * 1e-7 / (1 + atp)
    a4, b4 = 639.0 * atp / (1 + atp), 40.0 * rk ** 2 / di
    y1 = a4 * a1 * a2 + b2 * b4 * b3 + a2 * b4 * b3 + b3 * a1 * a2
    y2 = b2 * b1 * b4 + a1 * a2 * a3 + a3 * b1 * b4 + a2 * a3 * b4
    y3 = a2 * a3 * a4 + b3 * b2 * b1 + b2 * b1 * a4 + a3 * a4 * b1
    y4 = b4 * b3 * b2 + a3 * a4 * a1 + b2 * a4 * a1 + b3 * b2 * a1
    t = y1 + y2 + y3 + y4
    INaK = cls(30.0, 27.0, 21.0) * (3 * (y1 / t * a3 - y2 / t * b3) + 2 * (y4 / t * b1 - y3 / t * a1))
    # background
    IKb = cls(0.003, 0.0018, 0.003) * sg(-(v - 14.48) / 18.34) * (v - EK)
    INab = 3.75e-10 * vff * (nai * e1 - nao) / (e1 - 1)
    ICab = 2.5e-8 * 4 * vff * (cai * e2 - 0.341 * cao) / (e2 - 1)
    IpCa = 0.0005 * cai / (0.0005 + cai)
    dv = -(INa + INaL + Ito + ICaL + ICaNa + ICaK + IKr + IKs + IK1 + Ii + Iss + INaK + INab + IKb + IpCa + ICab + ist)
    vn = v + (dv + dvgap) * dt
    # fluxes and concentrations
    CaMKt = CaMKt + dt * (0.05 * CaMKb * (CaMKb + CaMKt) - 0.00068 * CaMKt)
    jn, jk, jc, jtr = (nass - nai) / 2, (kss - ki) / 2, (cass - cai) / 0.2, (cansr - cajsr) / 100
    den = 1 + (1.5 / cajsr) ** 8
    rel = cls(1.0, 1.0, 1.7) * -ICaL / den
    q = 4.75 / (1 + 0.0123 / cajsr)
    q, qp = where(q < 0.005, 0.0 * q + 0.005, q), where(1.25 * q < 0.005, 0.0 * q + 0.005, 1.25 * q)
    Jnp, Jp = relax(Jnp, 0.5 * 4.75 * rel, 1 / q), relax(Jp, 0.5 * 1.25 * 4.75 * rel, 1 / qp)
    Jrel = (1 - fP) * Jnp + fP * Jp
    upf = cls(1.0, 1.3, 1.0)
    Jup = (1 - fP) * upf * 0.004375 * cai / (cai + 0.00092) + fP * upf * 2.75 * 0.004375 * cai / (cai + 0.00075) - \
        0.0039375 * cansr / 15
    bi = 1 / (1 + cls(1.0, 1.3, 1.0) * 0.05 * 0.00238 / (0.00238 + cai) ** 2 + 0.07 * 0.0005 / (0.0005 + cai) ** 2)
    bs = 1 / (1 + 0.047 * 0.00087 / (0.00087 + cass) ** 2 + 1.124 * 0.0087 / (0.0087 + cass) ** 2)
    bj = 1 / (1 + 10.0 * 0.8 / (0.8 + cajsr) ** 2)
    dnai = -(INa + INaL + 3 * Ii + 3 * INaK + INab) * acap / (F * vmyo) + jn * vss / vmyo
    dnass = -(ICaNa + 3 * Iss) * acap / (F * vss) - jn
    dki = -(Ito + IKr + IKs + IK1 + IKb + ist - 2 * INaK) * acap / (F * vmyo) + jk * vss / vmyo
    dkss = -ICaK * acap / (F * vss) - jk
    dcai = bi * (-(IpCa + ICab - 2 * Ii) * acap / (2 * F * vmyo) - Jup * vnsr / vmyo + jc * vss / vmyo)
    dcass = bs * (-(ICaL - 2 * Iss) * acap / (2 * F * vss) + Jrel * vjsr / vss - jc)
    new = [vn, nai + dt * dnai, nass + dt * dnass, ki + dt * dki, kss + dt * dkss, cai + dt * dcai, cass + dt * dcass,
           cansr + dt * (Jup - jtr * vjsr / vnsr), cajsr + dt * bj * (jtr - Jrel), m, h, j, hsp, jp, mL, hL, hLp, a, iF,
           iS, ap, iFp, iSp, d, ff, fs, fcaf, fcas, jca, nca, ffp, fcafp, xrf, xrs, xs1, xs2, xk1, Jnp, Jp, CaMKt]
    return new, dv, (INa, ICaL, IKr, IKs, IK1)


REST = [-87.5, 7.0, 7.0, 145.0, 145.0, 1e-4, 1e-4, 1.2, 1.2, 0, 1, 1, 1, 1, 0, 1, 1, 0, 1, 1, 0, 1, 1, 0, 1, 1, 1, 1, 1,
        0, 1, 1, 0, 0, 0, 0, 1, 0, 0, 0]
T_REST, T_FINE, T_END = -40.0, 8.0, 460.0     # the beat's times relative to its stimulus, ms
FINE, COARSE = 0.1, 2.0                       # sampling of the beat in the upstroke and after it


@functools.lru_cache(maxsize=4)
def _beat(model):
    """One beat of endo, M and epi cells: [3, samples, 40] at -1 rest sample,
    every FINE ms up to T_FINE, every COARSE ms after; on the GPU."""
    par = MODELS[model][2]
    ct = np.array([ENDO, MID, EPI])
    s = [np.full(3, float(x)) for x in REST]
    with np.errstate(all="ignore"):
        for _ in range(int(-T_REST / 0.1)):
            s = _tpord(np, s, ct, par, 0.1, 0.0, 0.0)[0]
        out = [np.array(s).T]
        for i in range(int(round(T_FINE / DT))):
            s = _tpord(np, s, ct, par, DT, -52.0 if i * DT < 1.0 else 0.0, 0.0)[0]
            if (i + 1) % int(round(FINE / DT)) == 0:
                out.append(np.array(s).T)
        for i in range(int(round((T_END - T_FINE) / 0.1))):
            s = _tpord(np, s, ct, par, 0.1, 0.0, 0.0)[0]
            if (i + 1) % int(round(COARSE / 0.1)) == 0:
                out.append(np.array(s).T)
    return torch.from_numpy(np.stack(out, 1)).cuda()


def _states(model, types, t):
    """[n, 40] states at times t (ms after the stimulus) of the beat."""
    lib = _beat(model)
    nf = int(round(T_FINE / FINE))
    t = t.clamp(0.0, T_END - 1e-3)
    x = torch.where(t < T_FINE, t / FINE, nf + (t - T_FINE) / COARSE)
    i = x.floor().clamp(max=lib.shape[1] - 2)
    f = (x - i).unsqueeze(1)
    row = torch.where(types == EPI, 2, torch.where(types == MID, 1, 0))
    i = i.long()
    return torch.lerp(lib[row, i], lib[row, i + 1], f)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(2 * int(seed) + 1)


# ---- geometry (torch; the same on every machine) -------------------------------------
@functools.lru_cache(maxsize=3)
def _sheet(nx, ny, fibre):
    """(types [nx+2, ny+2], fibre or None, S1 mask, distance from the S1 edge in mm)."""
    t = np.full((nx + 2, ny + 2), EMPTY, np.uint8)
    xe, xm = round(0.30 * nx), round(0.65 * nx)
    t[1:1 + xe, 1:-1], t[1 + xe:1 + xm, 1:-1], t[1 + xm:nx + 1, 1:-1] = ENDO, MID, EPI
    s1 = np.zeros_like(t)
    s1[1:4, 1:-1] = 1
    f = None
    if fibre:
        ang = np.linspace(0.3, 1.2, ny + 2)[None, :] + 0.0 * t
        f = np.stack([np.cos(ang), np.sin(ang), 0.0 * ang], -1).astype(np.float32)
    x = torch.arange(1, nx + 1, device="cuda", dtype=torch.float64).unsqueeze(1).expand(nx, ny)
    return t, f, s1, (x * 0.15).reshape(-1)


@functools.lru_cache(maxsize=3)
def _shell(nx, nz):
    """Truncated ellipsoid shell on an nx x nx x nz grid at 0.2 mm, fibres +60
    to -60 degrees through the wall, an M-cell island, S1 at the apex."""
    dx = 0.2
    a1, c1 = 0.4 * nx * dx, 0.75 * nz * dx
    w = 0.4 * a1
    a0, c0, zb = a1 - w, c1 - w, 0.88 * nz * dx
    ax = torch.arange(nx, device="cuda", dtype=torch.float64) * dx
    px, py = (ax - nx * dx / 2).view(-1, 1, 1), (ax - nx * dx / 2).view(1, -1, 1)
    pz = (torch.arange(nz, device="cuda", dtype=torch.float64) * dx - zb).view(1, 1, -1)
    rr = px * px + py * py
    q1, q0 = rr / a1 ** 2 + pz * pz / c1 ** 2, rr / a0 ** 2 + pz * pz / c0 ** 2
    inside = (pz <= 0) & (q1 <= 1) & (q0 >= 1)
    inside[0], inside[-1], inside[:, 0], inside[:, -1], inside[:, :, 0], inside[:, :, -1] = (False,) * 6
    cells = inside.reshape(-1).nonzero().squeeze(1)
    gx, gy, gz = cells // (nx * nz), cells // nz % nx, cells % nz
    x, y, z = px.reshape(-1)[gx], py.reshape(-1)[gy], pz.reshape(-1)[gz]
    s1, s0 = q1.reshape(-1)[cells].sqrt(), q0.reshape(-1)[cells].sqrt()
    e = (s0 - 1) / ((s0 - 1) + (1 - s1) + 1e-30)
    del q1, q0, inside, rr
    am = a0 + 0.475 * w
    isl = (x - am) ** 2 + y ** 2 + (z + 0.4 * c1) ** 2 < (0.3 * a1) ** 2
    ty = torch.where(e < 0.3, ENDO, torch.where(e >= 0.65, EPI,
                                                torch.where(isl, MID, torch.where(e < 0.475, ENDO, EPI))))
    a, c = a0 + e * w, c0 + e * w
    n = torch.stack([x / a ** 2, y / a ** 2, z / c ** 2], 1)
    n = n / n.norm(dim=1, keepdim=True).clamp_min(1e-12)
    r = (x * x + y * y).sqrt().clamp_min(1e-9)
    circ = torch.stack([-y / r, x / r, 0 * x], 1)
    mer = torch.stack([-n[:, 2] * n[:, 0], -n[:, 2] * n[:, 1], 1 - n[:, 2] ** 2], 1)
    mer = mer / mer.norm(dim=1, keepdim=True).clamp_min(1e-9)
    al = (math.pi / 3 * (1 - 2 * e)).unsqueeze(1)
    fv = al.cos() * circ + al.sin() * mer
    fv = (fv / fv.norm(dim=1, keepdim=True).clamp_min(1e-9)).float()
    total = nx * nx * nz
    types = torch.full((total,), EMPTY, dtype=torch.uint8, device="cuda")
    types[cells] = ty.to(torch.uint8)
    fib = torch.zeros((total, 3), device="cuda")
    fib[cells] = fv
    apex = (x * x + y * y + (z + c1) ** 2).sqrt()
    m1 = torch.zeros(total, dtype=torch.uint8, device="cuda")
    m1[cells] = (apex < 0.08 * c1).to(torch.uint8)
    shp = (nx, nx, nz)
    return types.cpu().numpy().reshape(shp), fib.cpu().numpy().reshape(shp + (3,)), m1.cpu().numpy().reshape(shp), apex


def _tissue(case):
    """(types, fibre, s1, distance of each tissue voxel from the stimulus, dx, electrodes)."""
    if case["kind"] == "sheet":
        t, f, s1, far = _sheet(case["nx"], case["ny"], case["fibre"])
        return t, f, s1, far, 0.15, None
    t, f, s1, far = _shell(case["nx"], case["nz"])
    c, r = case["nx"] * 0.1, case["nx"] * 0.08 + 20.0
    el = [[c + r * math.cos(k * math.pi / 3), c + r * math.sin(k * math.pi / 3), case["nz"] * 0.1] for k in range(6)]
    return t, f, s1, far, 0.2, np.array(el) if case["ecg"] else None


def _protocol(case):
    """S1 inside the pass for the start-of-beat case, else long after it."""
    return dict(bcl=1000.0, s1_start=2.2 if case.get("s1") else 600.0, s1_duration=2.0, s1_strength=-52.0, s1_beats=0)


def _tissue_states(case, seed):
    """[n, 40] FP64 states: a wave from the stimulus site, `phase` ms after it
    started, its speed, phase and front shape a little different for every seed."""
    t, _, _, far, _, _ = _tissue(case)
    types = torch.from_numpy(t[t != EMPTY].reshape(-1)).cuda()
    u = torch.rand(4, generator=_gen(seed), device="cuda", dtype=torch.float64)
    k = torch.arange(len(types), device="cuda", dtype=torch.float64)
    wob = 0.4 * torch.sin(far * (0.5 + 0.3 * u[2]) + 6.283 * u[3] + k * (1e-4 * u[2]))
    tau = case["phase"] + 4.0 * (u[0] - 0.5) - far / (0.55 + 0.1 * u[1]) + wob
    s = _states("sheet" if case["kind"] == "sheet" else "shell", types, tau)
    s[:, 0] += 0.5 * torch.sin(far * 0.7 + 6.283 * u[3])
    return s, types


def _model(name):
    preset, kw, _ = MODELS[name]
    return lq.model(preset, **kw)


_scratch = {}


def _host(x):
    """A host copy through one pinned scratch buffer (valid until the next call)."""
    x = x.contiguous()
    b = _scratch.get("b")
    if b is None or b.numel() < x.numel():
        _scratch["b"] = b = torch.empty(x.numel(), dtype=torch.float64, pin_memory=True)
    b = b[:x.numel()]
    b.copy_(x.reshape(-1))
    return b.numpy().reshape(x.shape)


def _cell_inputs(case, seed):
    g = _gen(seed)
    n = case["n"]
    types = torch.tensor([ENDO, MID, EPI], device="cuda")[torch.randint(0, 3, (n,), device="cuda", generator=g)]
    t = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 440.0
    t[::4] *= 0.05                                   # a quarter around the upstroke
    dv = 0.05 * (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) - 0.5)
    return types, _states("cpu", types, t), dv


def _strand_types(n):
    ne, nm = round(0.25 * n), round(0.35 * n)
    return np.array([ENDO] * ne + [MID] * nm + [EPI] * (n - ne - nm), np.uint8)


def _batch_inputs(case, seed):
    """Per instance: types, model factors, stop time; and all states."""
    r = np.random.default_rng(case.get("instances", 0))       # the batch's make-up is the case's
    if case["kind"] == "strand":
        inst = [(_strand_types(case["n"]), MODELS["cpu"][2], case["ms"])]
    else:
        inst = []
        for _ in range(case["instances"]):
            ty = np.array([r.choice([ENDO, MID, EPI])], np.uint8) if r.random() < 0.5 else \
                _strand_types(int(r.integers(50, 401)))
            par = (1 - 0.95 * r.random(), r.uniform(1, 2), r.uniform(1, 2), 0.0, 0.0)
            inst.append((ty, par, case["ms"] * r.uniform(0.2, 1.0)))
    r = np.random.default_rng(seed)
    cv = 0.55 + 0.1 * r.random()
    tau = []
    for ty, _, _ in inst:
        x = np.arange(len(ty)) * 0.15
        tau.append(r.uniform(2.0, 380.0 if case["kind"] == "sweep" else 20.0) - x / cv)
    types = np.concatenate([i[0] for i in inst])
    s = _states("cpu" if case["kind"] == "strand" else "shell", torch.from_numpy(types).cuda(),
                torch.from_numpy(np.concatenate(tau)).cuda())
    return inst, types, s


def _train_inputs(case, seed):
    """Raw features, corrections, the mini-batches' rows, weights and norms."""
    g = _gen(seed)
    n = 200_000
    ty = torch.tensor([ENDO, MID, EPI], device="cuda")[torch.randint(0, 3, (n,), device="cuda", generator=g)]
    t = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 450.0
    s = _states("shell", ty, t)[:, surrogate.REF_INDEX].float()
    par = torch.rand(n, 3, generator=g, device="cuda") * torch.tensor([0.95, 1.2, 1.0], device="cuda") + \
        torch.tensor([0.05, 1.0, 1.0], device="cuda")
    hot = torch.stack([ty == ENDO, ty == EPI, ty == MID], 1).float()
    X = torch.cat([s * (1 + 0.01 * torch.randn(n, 38, generator=g, device="cuda")), par, hot], 1).contiguous()
    mu, sd = X.double().mean(0), X.double().std(0)
    mean, scale = np.zeros(48, np.float32), np.ones(48, np.float32)
    mean[:44], scale[:44] = mu.cpu(), (1 / sd.clamp_min(1e-9)).cpu()
    z = (X - mu.float()) / sd.clamp_min(1e-9).float()
    out = np.ones(48, np.float32)
    out[:38] = 1e-3 * np.exp(-np.arange(38) / 8)
    mix = torch.randn(44, 38, generator=g, device="cuda") / 6
    D = (torch.tanh(z @ mix) * torch.from_numpy(out[:38]).cuda()).contiguous()
    idx = torch.stack([torch.randint(0, n, (case["batch"],), generator=g, device="cuda") for _ in range(case["steps"])])
    return X, D, idx.contiguous(), _weights(g), (mean, scale, out)


def _weights(g):
    # W1 [128, 48], b1, W2 [128, 128], b2, W3 [48, 128], b3
    w = [torch.randn(n, generator=g, device="cuda") * s for n, s in (
        (6144, math.sqrt(2 / 48)), (128, 0.1), (16384, math.sqrt(2 / 128)), (128, 0.1), (6144, math.sqrt(1 / 128)),
        (48, 0.1))]
    return torch.cat(w).bfloat16().float()


# ---- prepare and run ------------------------------------------------------------------
def _whole_state(case):
    """Small tissues and the FP64 form are read back whole, the others' V."""
    return case["fp64"] or (case["kind"] == "sheet" and case["nx"] * case["ny"] <= 20000 and not case["readback"])


def _pinned(n, rows=None):
    return torch.empty((rows, n) if rows else n, dtype=torch.float32, pin_memory=True).numpy()


def prepare(case, seed):
    k, st = case["kind"], dict(case=case)
    if k == "cells":
        types, s, dv = _cell_inputs(case, seed)
        c = lq.TPORdCells(types.cpu().numpy().astype(np.uint8), precision=lq.FP64 if case["fp64"] else lq.MIXED)
        c.set_state(_host(s))
        c.set_dvgap_dt(dv.cpu().numpy())
        st.update(cells=c, ist=0.0 if case["n"] > 1 else -2.0)
    elif k in ("strand", "sweep"):
        inst, types, s = _batch_inputs(case, seed)
        models, specs = [], []
        for i, (ty, par, stop) in enumerate(inst):
            models.append(lq.model("baseline", gks_scale=par[0], pca_scale=par[1], gks_iso_scale=par[2],
                                   dss_shift=par[3], fss_shift=par[4]))
            specs.append(lq.InstanceSpec(types=ty, model=i, bcl=1000.0, s1_start=1.0, s1_duration=1.0, t_stop=stop,
                                         n_stim=min(3, len(ty)), record=k == "strand", ecg_x0=0.15 * len(ty) + 20.0))
        b = lq.Batch(specs, models, precision=lq.FP64 if case.get("fp64") else lq.MIXED, max_beats=4)
        b.set_state(_host(s))
        st.update(batch=b)
    elif k in ("sheet", "shell"):
        types, fibre, s1, _, dx, el = _tissue(case)
        sim = lq.Sim(types, dx, fibre=fibre, d_fibre=D_FIBRE, d_trans=D_TRANS, model=_model(k),
                     precision=lq.FP64 if case["fp64"] else lq.MIXED)
        sim.set_protocol(s1_mask=s1, **_protocol(case))
        sim.set_state(_host(_tissue_states(case, seed)[0]))
        if el is not None:
            sim.set_electrodes(el, every=50)
        if case["sur"]:
            sim.set_surrogate(_network())
        sim.step(2 if case["fp64"] else WARM)
        st.update(sim=sim)
        st["v"] = _pinned(sim.n, RING if case.get("readback") else None)
        if _whole_state(case):
            st["state"] = torch.empty((sim.n, 40), dtype=torch.float64, pin_memory=True).numpy()
    elif k == "train":
        X, D, idx, w, norm = _train_inputs(case, seed)
        m = lq.surrogate.Mlp(seed=1)
        m.set_norm(*norm)
        m.set_params(w.cpu().numpy())
        lib = _native.lib()
        lib.lqt_sur_prepare.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_int64] + [ctypes.c_void_p] * 2
        st.update(mlp=m, lib=lib, X=X, D=D, idx=idx,
                  xb=torch.empty((case["batch"], 48), dtype=torch.bfloat16, device="cuda"),
                  t=torch.empty((case["batch"], 48), dtype=torch.float32, device="cuda"))
    else:
        g = _gen(seed)
        m = lq.surrogate.Mlp(seed=1)
        m.set_params(_weights(g).cpu().numpy())
        st.update(mlp=m, x=torch.randn(case["rows"], 48, generator=g, device="cuda").bfloat16(),
                  y=torch.empty(case["rows"], 48, device="cuda"))
    return st


@functools.lru_cache(maxsize=1)
def _network():
    return lq.surrogate.load()


def _f32(x):
    """The mixed form keeps FP32 values: its FP64 read-backs as FP32."""
    return x.astype(np.float32)


def run(st):
    case, k = st["case"], st["case"]["kind"]
    if k == "cells":
        c = st["cells"]
        if case["n"] == 1:
            c.set_istim(st["ist"])
        c.update(case["steps"])
        out = dict(v=c.get_v(), currents=c.get_currents()) if case["n"] == 1 else \
            dict(state=c.get_state())
        return out if case["fp64"] else {q: _f32(x) for q, x in out.items()}
    if k in ("strand", "sweep"):
        b = st["batch"]
        b.run()
        out = dict(state=b.get_state())
        if k == "strand":
            r = b.record(0)
            out.update(v=r["v"], ecg=r["ecg"])
        if not case.get("fp64"):
            out = {q: _f32(x) for q, x in out.items()}
        out["t_act"] = b.detect()["t_act"]
        return out
    if k in ("sheet", "shell"):
        sim = st["sim"]
        if case.get("readback") and not case["fp64"]:
            last = 0
            for i in range(case["steps"]):
                sim.step_async(1)
                if i >= RING:
                    sim.wait_v(last - RING + 1)
                last = sim.get_v_async(st["v"][i % RING])
            sim.wait_v()
            return dict(v=st["v"][:min(case["steps"], RING)])
        sim.step(case["steps"])
        if case["fp64"]:
            return dict(state=sim.get_state(out=st["state"]))
        if _whole_state(case):
            return dict(state=_f32(sim.get_state(out=st["state"])), t_act=sim.detect()["t_act"])
        sim.get_v_into(st["v"])
        return dict(v=st["v"], ecg=_f32(sim.ecg()[0])) if case.get("ecg") else dict(v=st["v"])
    if k == "train":
        m, lib, xb, t, n = st["mlp"], st["lib"], st["xb"], st["t"], case["batch"]
        loss = 0.0
        for i in range(case["steps"]):
            _native.check(lib.lqt_sur_prepare(m._h, st["X"].data_ptr(), st["D"].data_ptr(), st["idx"][i].data_ptr(), n,
                                              xb.data_ptr(), t.data_ptr()), "lqt_sur_prepare")
            if i + 1 < case["steps"]:
                _native.check(m.L.lqt_mlp_train_step(m._h, xb.data_ptr(), t.data_ptr(), n, 1e-3, None),
                              "lqt_mlp_train_step")
            else:
                loss = m.train_step(xb, t, 1e-3)
        return dict(params=m.params(), loss=np.float32(loss))
    st["mlp"].infer(st["x"], st["y"])
    return st["y"]


# ---- what a pass cannot do without ----------------------------------------------------
CELL_OPS = 1200          # arithmetic of one TPORd update, an exponential or a division counted once


def _count(case):
    """Cells and cell-steps of a pass."""
    k = case["kind"]
    if k == "cells":
        return case["n"], case["n"] * case["steps"]
    if k == "strand":
        return case["n"], case["n"] * (case["ms"] / DT + 1)
    if k == "sweep":
        c = case["instances"] * (0.5 + 0.5 * 225)
        return c, c * 0.6 * case["ms"] / DT
    if k == "sheet":
        return case["nx"] * case["ny"], case["nx"] * case["ny"] * case["steps"]
    a1, c1 = 0.08 * case["nx"], 0.15 * case["nz"]
    w = 0.4 * a1
    n = 2 / 3 * math.pi * (a1 * a1 * c1 - (a1 - w) ** 2 * (c1 - w)) / 0.008
    return n, n * case["steps"]


def work(case):
    k = case["kind"]
    if k == "train":
        macs = 48 * 128 + 128 * 128 + 128 * 48
        return dict(bytes=case["steps"] * case["batch"] * (44 + 38) * 4.0 + 8 * 4 * (macs + 304),
                    flops=6.0 * macs * case["batch"] * case["steps"])
    if k == "infer":
        return dict(bytes=case["rows"] * (96.0 + 192.0), flops=2.0 * (48 * 128 + 128 * 128 + 128 * 48) * case["rows"])
    n, steps = _count(case)
    state = 40 * (8 if case.get("fp64") else 4) + (0 if case.get("fp64") else 32)
    ops = CELL_OPS
    by = 2.0 * n * state + 16 * n
    if case.get("sur"):                    # every tenth step the network and the coarse step, diffusion on all
        ops = 60 + (CELL_OPS + 57344) / 10
    if case.get("readback"):
        by += 4.0 * steps
    return dict(bytes=by, flops=float(ops) * steps)


# ---- 64-bit results ---------------------------------------------------------------------
_IC3 = ((3, 3, 1), (1, 3, -1), (6, 2, 1), (9, 3, 1), (7, 3, -1), (4, 2, -1), (12, 2, 1), (10, 2, -1), (14, 1, 1),
        (17, 2, 1), (15, 2, -1), (13, 1, -1), (20, 3, 1), (18, 3, -1), (23, 2, 1), (26, 3, 1), (24, 3, -1), (21, 2, -1))
_IR3 = ((9, 3, 1), (2, 2, -1), (3, 3, -1), (1, 3, -1), (8, 2, 1), (7, 3, 1), (17, 2, 1), (11, 1, -1), (12, 2, -1),
        (10, 2, -1), (16, 1, 1), (15, 2, 1), (26, 3, 1), (19, 2, -1), (20, 3, -1), (18, 3, -1), (25, 2, 1), (24, 3, 1))
_IL3 = ((18, 3, 1), (19, 2, 1), (20, 3, 1), (21, 2, 1), (22, 1, 1), (23, 2, 1), (24, 3, 1), (25, 2, 1), (26, 3, 1),
        (1, 3, -1), (2, 2, -1), (3, 3, -1), (4, 2, -1), (5, 1, -1), (6, 2, -1), (7, 3, -1), (8, 2, -1), (9, 3, -1))


def _mirror(shape, tissue):
    """Empty voxels beside tissue and the tissue voxel each mirrors: the
    neighbour nearest to the occupancy normal (GPU3D.cu:1487-1604); on a
    rectangular sheet that is the edge or corner voxel it touches."""
    nx, ny, nz = shape
    grid = tissue.view(shape)
    if nz == 1:
        g = torch.nonzero(~tissue).squeeze(1)
        x, y = (g // ny).clamp(1, nx - 2), (g % ny).clamp(1, ny - 2)
        return g, x * ny + y
    pad = torch.zeros((nx + 2, ny + 2, nz + 2), dtype=torch.bool, device="cuda")
    pad[1:-1, 1:-1, 1:-1] = grid
    offs = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1) if (a, b, c) != (0, 0, 0)]
    near = torch.zeros(shape, dtype=torch.bool, device="cuda")
    for a, b, c in offs:
        near |= pad[1 + a:1 + a + nx, 1 + b:1 + b + ny, 1 + c:1 + c + nz]
    g = torch.nonzero((near & ~grid).view(-1)).squeeze(1)
    x, y, z = g // (ny * nz), g // nz % ny, g % nz

    def at(a, b, c):
        return pad[x + 1 + a, y + 1 + b, z + 1 + c]

    occ = [None] + [at(*o).double() for o in offs]
    div = (None, 1.0, math.sqrt(2.0), math.sqrt(3.0))

    def total(terms):
        s = torch.zeros(len(g), dtype=torch.float64, device="cuda")
        for slot, kind, sign in terms:
            s = s + sign * (occ[slot] / div[kind])
        return s

    ic, ir, il = total(_IC3), total(_IR3), total(_IL3)
    big = torch.maximum(torch.maximum(ic.abs(), ir.abs()), il.abs())
    flat = big < 0.0001
    nv = [torch.where(flat, 0.0 * q, q / big) for q in (il, ir, ic)]
    best = torch.full((len(g),), 1000.0, dtype=torch.float64, device="cuda")
    src = g.clone()
    for zc in (-1, 0, 1):
        for yc in (-1, 0, 1):
            for xc in (-1, 0, 1):
                dis = ((xc - nv[0]) * (xc - nv[0]) + (yc - nv[1]) * (yc - nv[1]) + (zc - nv[2]) * (zc - nv[2])).sqrt()
                hit = at(xc, yc, zc) & (dis < best)
                best = torch.where(hit, dis, best)
                src = torch.where(hit, ((x + xc) * ny + y + yc) * nz + z + zc, src)
    return g, src


def _exact_tissue(case, seed):
    types, fibre, s1, _, dx, el = _tissue(case)
    shape = types.shape + (1,) * (3 - types.ndim)
    nx, ny, nz = shape
    tissue = torch.from_numpy(types.reshape(-1) != EMPTY).cuda()
    cells = torch.nonzero(tissue).squeeze(1)
    n = len(cells)
    s, ct = _tissue_states(case, seed)
    s = [s[:, i].clone() for i in range(40)]
    dst, src = _mirror(shape, tissue)
    V = torch.zeros(nx * ny * nz, dtype=torch.float64, device="cuda")
    sx, sy = ny * nz, nz
    S1 = torch.from_numpy(s1.reshape(-1)).cuda()[cells].bool()
    pr = _protocol(case)
    D = B = None
    if fibre is not None:
        f = torch.from_numpy(fibre.reshape(-1, 3)).cuda()[cells].double()
        dd = D_FIBRE - D_TRANS
        of = torch.full((nx * ny * nz,), -1, dtype=torch.long, device="cuda")
        of[cells] = torch.arange(n, device="cuda")
        D = {}
        for i in range(3):
            for j in range(i, 3):
                D[i, j] = D[j, i] = dd * f[:, i] * f[:, j] + (D_TRANS if i == j else 0.0)
        B = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
        for i, stride in ((0, sx), (1, sy), (2, 1)):
            if shape[i] == 1:
                continue
            p, m = of[cells + stride], of[cells - stride]
            for j in range(3):
                q = D[i, j]
                hi, lo = torch.where(p >= 0, q[p.clamp_min(0)], q), torch.where(m >= 0, q[m.clamp_min(0)], q)
                steps = ((p >= 0).double() + (m >= 0).double()).clamp_min(1.0)
                B[j] += (hi - lo) / (steps * dx)
    # the path stores the tensor in 32 bits; these are its 64-bit values
    time, echo, vs = 0.0, [], []
    warm = 2 if case["fp64"] else WARM
    act = torch.full((n,), -1.0, dtype=torch.float64, device="cuda")
    par = MODELS[case["kind"]][2]
    for k in range(warm + case["steps"]):
        V[cells] = s[0]
        V[dst] = V[src]
        vc = s[0]

        def at(o):
            return V[cells + o]

        xp_, xm_, yp, ym = at(sx), at(-sx), at(sy), at(-sy)
        lxx, lyy = (xp_ + xm_ - 2 * vc) / dx ** 2, (yp + ym - 2 * vc) / dx ** 2
        if nz > 1:
            zp, zm = at(1), at(-1)
            lzz = (zp + zm - 2 * vc) / dx ** 2
        if D is None:
            du = D_FIBRE * (lxx + lyy + (lzz if nz > 1 else 0.0))
        else:
            c4 = 4 * dx ** 2
            lxy = (at(sx + sy) + at(-sx - sy) - at(-sx + sy) - at(sx - sy)) / c4
            du = D[0, 0] * lxx + D[1, 1] * lyy + 2 * D[0, 1] * lxy + (B[0] * (xp_ - xm_) + B[1] * (yp - ym)) / (2 * dx)
            if nz > 1:
                lxz = (at(sx + 1) + at(-sx - 1) - at(-sx + 1) - at(sx - 1)) / c4
                lyz = (at(sy + 1) + at(-sy - 1) - at(-sy + 1) - at(sy - 1)) / c4
                du = du + D[2, 2] * lzz + 2 * (D[0, 2] * lxz + D[1, 2] * lyz) + B[2] * (zp - zm) / (2 * dx)
        on = pr["s1_start"] <= time < pr["s1_start"] + pr["s1_duration"]
        ist = torch.where(S1, pr["s1_strength"], 0.0).double() if on else 0.0
        new = _tpord(torch, s, ct, par, DT, ist, du)[0]
        if time >= pr["s1_start"]:
            hit = (vc < -30.0) & (new[0] >= -30.0) & (act < 0)
            act = torch.where(hit, torch.full_like(act, time), act)
        s = new
        time += DT
        if k >= warm:
            vs.append(s[0])
            vs = vs[-RING:] if case.get("readback") else vs[-1:]
        if el is not None and (k + 1) % 50 == 0:
            V[cells] = s[0]
            V[dst] = V[src]
            h = [(at(o) - at(-o)) / 2 for o in (sx, sy, 1)]
            pos = torch.stack([cells // sx, cells // nz % ny, cells % nz], 1).double() * dx
            echo.append(torch.stack([sum(h[i] * (pos[:, i] - e[i]) for i in range(3)).div(
                sum((pos[:, i] - e[i]) ** 2 for i in range(3)) ** 1.5).sum() for e in el]))
    if case["fp64"]:
        return dict(state=torch.stack(s, 1))
    if case.get("readback"):
        ring = [None] * min(case["steps"], RING)
        for i, v in enumerate(vs, max(0, case["steps"] - RING)):
            ring[i % RING] = v
        return dict(v=torch.stack(ring))
    if _whole_state(case):
        return dict(state=torch.stack(s, 1), t_act=act)
    return dict(v=s[0], ecg=torch.stack(echo)) if el is not None else dict(v=s[0])


def _exact_cells(case, seed):
    types, s, dv = _cell_inputs(case, seed)
    ist = 0.0 if case["n"] > 1 else -2.0
    small = case["n"] < 4000 and not (case["n"] > 64 and case["steps"] > 500)
    xp, ct = (np, types.cpu().numpy()) if small else (torch, types)
    s = [q.cpu().numpy() if small else q.clone() for q in s.T]
    dv = dv.cpu().numpy() if small else dv
    d = cur = None
    with np.errstate(all="ignore"):
        for _ in range(case["steps"]):
            s, d, cur = _tpord(xp, s, ct, MODELS["cpu"][2], DT, ist, dv)
    cur = list(cur) + [abs(d)]
    stack = np.stack if small else torch.stack
    return dict(v=s[0], currents=stack(cur, 1)) if case["n"] == 1 else dict(state=stack(s, 1))


def _exact_batch(case, seed):
    inst, types, s = _batch_inputs(case, seed)
    big = len(types) > 4000
    xp = torch if big else np
    lens = np.array([len(i[0]) for i in inst])
    first = np.concatenate([[0], np.cumsum(lens)[:-1]])
    li = np.concatenate([np.arange(q) for q in lens])
    own = np.arange(len(types))
    left, right = np.where(li > 0, own - 1, own), np.where(li < np.repeat(lens, lens) - 1, own + 1, own)
    stop = np.zeros(len(inst), np.int64)
    axis, t = [], 0.0
    while t <= max(i[2] for i in inst):
        axis.append(t)
        t += DT
    for i, q in enumerate(inst):
        stop[i] = np.searchsorted(axis, q[2], side="right")
    arr = (lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()) if big else (lambda x: x)
    par = [arr(np.repeat(np.array([i[1][j] for i in inst]), lens)) for j in range(5)]
    ends, stim = arr(np.repeat(stop, lens)), arr(li < 3)
    L, Rr, ct = arr(left), arr(right), arr(types.astype(np.int64))
    coef = arr(np.where(np.repeat(lens, lens) > 1, 0.154 / 0.15 ** 2, 0.0))
    s = [q.clone() if big else q.cpu().numpy() for q in s.T]
    act = 0.0 * s[0] - 1.0
    rec, ecg, opened = [], [], False
    with np.errstate(all="ignore"):
        for k, t in enumerate(axis):
            v = s[0]
            on = 1.0 <= t < 2.0
            ist = xp.where(stim, -52.0 + 0.0 * v, 0.0 * v) if on else 0.0
            new = _tpord(xp, s, ct, par, DT, ist, coef * (v[L] + v[Rr] - 2 * v))[0]
            go = ends > k
            s = [xp.where(go, a, b) for a, b in zip(new, s)] if k >= stop.min() else new
            opened |= on
            if opened:
                act = xp.where(go & (act < 0) & (v < -30.0) & (s[0] >= -30.0), 0.0 * v + t, act)
            if case["kind"] == "strand" and k % 10 == 0:
                rec.append(s[0])
                g = np.gradient(s[0])
                ecg.append(np.sum(-g / (own * 0.15 - (0.15 * len(own) + 20.0)) ** 2))
    st = torch.stack(s, 1) if big else np.stack(s, 1)
    acts = None if case["kind"] == "sweep" else np.stack([act] + [0 * act - 1] * 3, 1)
    out = dict(state=st, t_act=acts)
    if case["kind"] == "strand":
        out.update(v=np.stack(rec), ecg=np.array(ecg))
    return out


def _exact_train(case, seed):
    X, D, idx, w, (mean, scale, out) = _train_inputs(case, seed)
    up = lambda a: torch.from_numpy(a).cuda().double()  # noqa: E731
    mean, scale, out = up(mean), up(scale), up(out)
    p = w.double()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    size, loss = case["batch"], None
    for k in range(case["steps"]):
        x = torch.zeros(size, 48, dtype=torch.float64, device="cuda")
        x[:, :44] = (X[idx[k]].double() - mean[:44]) * scale[:44]
        t = D[idx[k]].double() / out[:38]
        w1, b1, w2, b2, w3, b3 = (q.view(sh) for q, sh in zip(
            p.split([6144, 128, 16384, 128, 6144, 48]), ((128, 48), (128,), (128, 128), (128,), (48, 128), (48,))))
        z1 = x @ w1.T + b1
        h1 = z1 * z1.sigmoid()
        z2 = h1 @ w2.T + b2
        h2 = z2 * z2.sigmoid()
        y = h2 @ w3.T + b3
        r = y.clone()
        r[:, :38] -= t
        r[:, 38:] = 0
        loss = float((r ** 2).sum() / (size * 38))
        dy = 2 * r / (size * 38)
        d2 = (dy @ w3) * (z2.sigmoid() * (1 + z2 * (1 - z2.sigmoid())))
        d1 = (d2 @ w2) * (z1.sigmoid() * (1 + z1 * (1 - z1.sigmoid())))
        g = torch.cat([q.reshape(-1) for q in (d1.T @ x, d1.sum(0), d2.T @ h1, d2.sum(0), dy.T @ h2, dy.sum(0))])
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - 1e-3 * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return dict(params=p, loss=loss)


def exact(case, seed):
    k = case["kind"]
    if k == "cells":
        return _exact_cells(case, seed) if case["steps"] <= 2000 else None
    if k in ("strand", "sweep"):
        return _exact_batch(case, seed)
    if k in ("sheet", "shell"):
        return _exact_tissue(case, seed) if _count(case)[0] * (WARM + case["steps"]) < 6e8 else None
    if k == "train":
        return _exact_train(case, seed)
    g = _gen(seed)
    p = _weights(g).double()
    x = torch.randn(case["rows"], 48, generator=g, device="cuda").bfloat16().double()
    w1, b1, w2, b2, w3, b3 = (q.view(sh) for q, sh in zip(
        p.split([6144, 128, 16384, 128, 6144, 48]), ((128, 48), (128,), (128, 128), (128,), (48, 128), (48,))))
    z = x @ w1.T + b1
    z = (z * z.sigmoid()) @ w2.T + b2
    return (z * z.sigmoid()) @ w3.T + b3
