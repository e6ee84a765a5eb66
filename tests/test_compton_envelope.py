"""The early rejection of GCOa's trials (compton_refused).

A trial is rejected when u * s0 > s(theta) * T(tau); the envelope part rejects
it already when u > 1.001 * T(tau), which is the same answer as long as the
shell sum s never exceeds s0 by 0.1 % and T is the same number in both parts.

The sum, on the CPU with the formula in numpy: s grows with theta (each shell's
projected momentum does: d pz / d aux has the sign of aux + u^2 + u m c^2) and
s0 is its value at pi, so only the rounding of the two single-precision sums
can exceed it: each of at most 30 terms is off by a few units of 2^-24 of the
sum plus the exponential's 2^-22, below 1e-5 together.  Checked on every staged
material at random energies and angles, the smallest and the backward ones
among them, with half of the margin.

T, on the GPU with the library's two parts: its numerator cancels to about
ek^2 (1e-4 at 5 keV), where two ways to round it differ by up to 0.13 %, more
than the margin.  No trial that the early part rejects is one that the whole
test accepts, with draws close to T and close to the early part's line."""
import numpy as np
import pytest

import mcpet
from mcpet import inputs
import scenes

MC2, INV_MC2, R2, IR2 = (np.float32(x) for x in (510998.918, 1.956951306108245e-6, 1.4142135623731, 0.70710678118654502))


def _sum(E, cdt1, mat, t):
    """Shell sum at 1 - cos(theta) = cdt1 in the device formula's precision."""
    s = np.zeros_like(E)
    half, one = np.float32(0.5), np.float32(1)
    for i in range(int(t["noscco"][mat])):
        u, f, j = (np.float32(t[k][mat + i * 15]) for k in ("uico", "fco", "fj0"))
        on = u < E
        aux = E * (E - u) * cdt1
        pz = j * (aux - u * MC2) / np.sqrt(np.where(on, aux + aux + u * u, one)) * INV_MC2
        pz = np.where((aux > 1e-12) | (u > 1e-12), pz, np.float32(0.002))
        a = np.abs(pz) * R2 + IR2
        term = half * np.exp(half - a * a)
        s = s + np.where(on, f * np.where(pz > 0, one - term, term), np.float32(0))
    return s


@pytest.mark.parametrize("extended", [False, True], ids=["5-515keV", "5-1250keV"])
def test_no_shell_sum_exceeds_the_normaliser(workdir, extended):
    mat, rho, act, vs, used = inputs.head_phantom(shape=(12, 24, 24), voxel_cm=1.0, seed=5, total_bq=1e4)
    sc = scenes.scene_from_arrays(workdir, mat, rho, act, vs, tissues=used, extended=extended,
                                  **inputs.scanner_for_head())
    t, info = sc.export_tables(), sc.info
    top = float(info.e0) + (int(info.n_energy) - 1) / float(info.inv_de)
    rng = np.random.default_rng(3)
    n = 400_000
    E = rng.uniform(float(info.e0), top, n).astype(np.float32)
    cdt1 = np.concatenate([rng.uniform(0, 2, n // 2), 10.0 ** rng.uniform(-9, 0, n // 4),
                           2 - 10.0 ** rng.uniform(-7, -1, n - n // 2 - n // 4)]).astype(np.float32)
    checked = 0
    for m in range(15):
        if t["noscco"][m] <= 0:
            continue
        s, s0 = _sum(E, cdt1, m, t), _sum(E, np.full(n, 2, np.float32), m, t)
        assert np.all(s <= np.float32(1.0005) * s0), f"material {m}"
        checked += 1
    assert checked >= 2
    sc.close()


def _fma(a, b, c):
    """a * b + c rounded once (a product of two floats is exact in double)."""
    return (a.astype(np.float64) * b + c).astype(np.float32)


def _factor(E, tau):
    """Numerator and denominator of T as compton_factor rounds them."""
    ek = E * INV_MC2
    ek2, ek3 = ek * np.float32(2) + np.float32(1), ek * ek
    inner = _fma(tau, ek2 + tau * ek3, (ek3 - ek2) - np.float32(1))
    return _fma(tau, inner, 1.0), ek3 * tau * _fma(tau, tau, 1.0)


@pytest.mark.gpu
@pytest.mark.parametrize("low, high, backward", [(5e3, 5.5e3, True), (5.5e3, 8e3, True), (5e3, 20e3, False),
                                                 (20e3, 511e3, False)],
                         ids=["5-5.5keV-backward", "5.5-8keV-backward", "5-20keV", "20-511keV"])
def test_no_early_rejection_of_an_accepted_draw(workdir, low, high, backward):
    mat, rho, act, vs, used = inputs.head_phantom(shape=(12, 24, 24), voxel_cm=1.0, seed=5, total_bq=1e4)
    sc = scenes.scene_from_arrays(workdir, mat, rho, act, vs, tissues=used, **inputs.scanner_for_head())
    mats = [m for m in range(15) if sc.export_tables()["noscco"][m] > 0]
    rng = np.random.default_rng(int(low))
    n, bad, early_kept, early_refused = 8_000_000, 0, 0, 0
    for k in range(4):
        e = rng.uniform(low, high, n).astype(np.float32)
        ek = e.astype(np.float64) / 510998.918
        cdt1 = 2 - 10.0 ** rng.uniform(-6, -2, n) if backward else rng.uniform(0, 2, n)
        tau = (1 / (1 + ek * cdt1)).astype(np.float32)
        num, den = _factor(e, tau)
        # half the draws around the factor in the device's rounding, where only another rounding can reject
        # early, half around the early part's line
        near = np.where(np.arange(n) & 1, rng.uniform(0.9995, 1.0001, n), rng.uniform(1.0005, 1.0015, n))
        u = (num.astype(np.float64) / den * near).astype(np.float32)
        early, whole = mcpet.probe_compton_test(sc, e, rng.choice(mats, n), tau, u)
        bad += int((early & ~whole).sum())
        early_kept += int((~early).sum())
        early_refused += int(early.sum())
    sc.close()
    assert min(early_kept, early_refused) > n // 2         # the draws lie on both sides of the line
    assert bad == 0
