"""The early rejection of GCOa's trials (compton_envelope).

A trial is rejected when u * s0 > s(theta) * T(tau); the envelope part rejects
it already when u > 1.001 * T(tau), which is the same answer as long as the
shell sum s never exceeds s0 by 0.1 %.  s grows with theta (each shell's
projected momentum does: d pz / d aux has the sign of aux + u^2 + u m c^2) and
s0 is its value at pi, so only the rounding of the two single-precision sums
can: each of at most 30 terms is off by a few units of 2^-24 of the sum plus
the exponential's 2^-22, below 1e-5 together.  Checked on every staged
material at random energies and angles, the smallest and the backward ones
among them, with half of the margin."""
import numpy as np
import pytest

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
