"""The FP64 digits' low-order parts, which a comparison with FP64 multiply-adds cannot see: eigenvalues of the seeded runs
against the same runs in extended precision (numpy's long double: at least 64 bits), the FP32 normals recovered from
the exported increments (dB = z / sqrt(T), one rounding in FP64, so that rounding dB sqrt(T) to FP32 gives z back).

Tolerance: the form's stated rms error at dim 12 (csrc/jne_accum_digits.cuh: 7.8e-15 at T 1000, 9.3e-15 at T 10^4) times
five, which covers the other models' larger conditioning.  Without the last sum G_5 the digits' own error, emulated in
integers on 16 runs, is 9e-14 (dim 4, T 2100) to 4e-12 (dim 12, T 33) at these shapes, with it 1.3e-15 to 1e-14."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _eigs(z, model):
    """Descending eigenvalues of the pencil of (runs, T, dim) normals, B = W / sqrt(T)."""
    z = z.astype(LD)
    runs, T, dim = z.shape
    W = np.zeros_like(z)
    W[:, 1:] = np.cumsum(z, axis=1)[:, :-1]
    y = np.broadcast_to((np.arange(1, T + 1, dtype=LD) / T)[None, :, None], (runs, T, 1))
    one = np.ones_like(y)
    if model == 0:
        F = W
    elif model == 1:
        F = np.concatenate([W, one], axis=2)
    elif model in (2, 3):
        rows = W[:, :, :dim - 1] if model == 2 else W
        F = np.concatenate([rows - rows.mean(axis=1, keepdims=True), y - LD(0.5)], axis=2)
    else:
        F = np.concatenate([W[:, :, :dim - 1], y * y], axis=2)
        for q in (one, y - y.mean(axis=1, keepdims=True)):  # orthogonal to each other
            F = F - q * (F * q).sum(axis=1, keepdims=True) / (q * q).sum(axis=1, keepdims=True)
    k = F.shape[2]
    S11, E = np.einsum("rta,rtb->rab", F, F), np.einsum("rtc,rta->rca", z, F)
    L = np.zeros_like(S11)
    for j in range(k):  # Cholesky, then E = S10 L^-T column by column
        for i in range(j + 1):
            s = S11[:, j, i] - (L[:, j, :i] * L[:, i, :i]).sum(axis=1)
            L[:, j, i] = np.sqrt(s) if i == j else s / L[:, i, i]
    for j in range(k):
        E[:, :, j] = (E[:, :, j] - (E[:, :, :j] * L[:, None, j, :j]).sum(axis=2)) / L[:, j, j][:, None]
    C = np.einsum("rca,rcb->rab", E, E)
    for _ in range(12):  # cyclic Jacobi
        for p in range(k):
            for q in range(p + 1, k):
                a = np.where(C[:, p, q] == 0, LD(1), C[:, p, q])
                th = (C[:, q, q] - C[:, p, p]) / (2 * a)
                t = np.where(th >= 0, 1, -1) / (np.abs(th) + np.hypot(th, LD(1)))
                t = np.where(C[:, p, q] == 0, LD(0), t)
                c = 1 / np.hypot(t, LD(1))
                s = t * c
                for ax in (1, 2):
                    M = np.moveaxis(C, ax, 2)
                    x, v = M[:, :, p].copy(), M[:, :, q].copy()
                    M[:, :, p], M[:, :, q] = c[:, None] * x - s[:, None] * v, s[:, None] * x + c[:, None] * v
    return -np.sort(-np.abs(np.einsum("rkk->rk", C)), axis=1)


@pytest.mark.parametrize("dim,steps", [(12, 33), (12, 500), (12, 1000), (12, 2500), (5, 700), (4, 2100)])
def test_against_extended_precision(engine, jne, dim, steps):
    runs = 32
    dB, _ = engine.export_increments(dim, steps, 5, runs)
    z = (dB * np.sqrt(steps)).astype(np.float32)
    for model in (0, 1, 3):
        ref = _eigs(z, model)
        got = engine.eigs_seeded(model, dim, steps, 5, runs, precision=jne.PREC_FP64)
        err = np.abs(got - ref).max(axis=1) / ref.max(axis=1)
        assert np.sqrt(np.mean(err**2)) < 4e-14, (model, float(np.sqrt(np.mean(err**2))))
