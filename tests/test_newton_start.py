"""The wall model's Newton iteration (csrc/physics.cuh spalding_utau) with its own start, its one
division and its stop after an update of 1e-9, restated here in NumPy scalar arithmetic: the
iterate it returns is the one of the reference's full iteration (wmles/wall_model.py:19-40) to
the rounding of its residual, and the settled flag is the same."""
import numpy as np
import pytest

KAPPA, B = 0.41, 5.2
EKB = np.exp(-KAPPA * B)
EPS = np.finfo(float).eps


def _reference(Reh, n):
    up, last = min(max(np.sqrt(Reh), 1.0), 25.0), 0.0
    for _ in range(n):
        ku = KAPPA * up
        ex = np.exp(ku)
        F = up + EKB * (ex - 1.0 - ku - 0.5 * ku * ku - ku * ku * ku / 6.0) - Reh / up
        dF = 1.0 + EKB * KAPPA * (ex - 1.0 - ku - 0.5 * ku * ku) + Reh / (up * up)
        nx = min(max(up - F / dF, 0.5 * up), 100.0)
        last, up = nx - up, nx
    return up, not (abs(last) <= 1e-8 * up)


def _device(Reh, n):
    up, last = min(max(np.sqrt(Reh), 1.0), 25.0), 0.0
    if n >= 30 and 625.0 < Reh < 1e12:
        up = min(max(np.log(Reh / (18.0 * EKB)) / KAPPA, 1.0), 100.0)
    for _ in range(n):
        ku = KAPPA * up
        ex = np.exp(ku)
        g = ex - 1.0 - ku - 0.5 * ku * ku
        num = (up + EKB * (g - ku * ku * ku * (1.0 / 6.0))) * up - Reh
        den = (1.0 + EKB * KAPPA * g) * (up * up) + Reh
        nx = min(max(up - num * up / den, 0.5 * up), 100.0)
        last, up = nx - up, nx
        if abs(last) <= 1e-9 * up:
            return up, False
    return up, not (abs(last) <= 1e-8 * up)


@pytest.mark.parametrize("n", (30, 29, 12, 4, 1, 0))
def test_start_and_stop_return_the_reference_iterate(n):
    rng = np.random.default_rng(3)
    Rehs = np.concatenate([10 ** rng.uniform(-1, 8, 3000), [1e-3, 1.0, 624.999, 625.0, 625.001, 1e7, 1e11, 2e12]])
    for Reh in Rehs:
        up, moving = _device(Reh, n)
        ref, ref_moving = _reference(Reh, n)
        assert moving == ref_moving, (Reh, n)
        # both iterates carry the rounding of F: some ten terms, the largest e^ku <= ekb^-1 (F + ...), each
        # with a unit in the last place (and exp one more), divided by u+ dF >= F's terms: 16 eps each;
        # an iterate that has not settled carries the rounding of up to n steps, each contracting
        assert abs(up - ref) <= 32 * EPS * ref, (Reh, n, up, ref)
