"""Sums over FP32 vectors in the mixed-precision solvers (csrc/solve.cu): |r|^2 of a vector that does not fill the
machine is the FP64 sum of exact products. A diagonal matrix of powers of two and an identity preconditioner make the
first iteration's residual known to the last bit, repeated in fours so that FP32 runs of four products would all be
rounded the same way, and the inner tolerance is put halfway between the two sums (5e-9 apart at least; the FP64 sum
itself is good to 1e-13): the iteration at which the inner solve stops tells which one was taken."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32, f64 = np.float32, np.float64
D4 = np.array([1.0, 2.0, 0.5, 4.0])


def _first_iteration(b4, n):
    """|r|^2 / |r0|^2 after one iteration, summed in FP64 and in FP32 runs of four."""
    k = n // 4
    s = 1.0 / np.sqrt(k * float((b4 * b4).sum()))
    r = (b4 * s).astype(f32)
    rr0 = float((r.astype(f64) ** 2).sum())
    pAp = float(((D4.astype(f32) * r) * r).astype(f64).sum())
    al = f32(rr0 / pAp)
    Ap = D4.astype(f32) * r
    r1 = (r.astype(f64) - f64(al) * Ap.astype(f64)).astype(f32)  # one rounding, as a fused multiply-add
    exact = float((r1.astype(f64) ** 2).sum())
    run = f32(0)
    for v in r1:
        run = f32(f64(run) + f64(v) * f64(v))
    return exact / rr0, float(run) / rr0


def _pattern(n, want_above):
    rng = np.random.default_rng(n)
    for _ in range(10000):
        b4 = rng.integers(1, 4096, 4).astype(f64)
        e, r = _first_iteration(b4, n)
        if (r > e) == want_above and abs(r - e) > 2e-8 * e:
            return b4, np.sqrt(0.5 * (e + r))
    raise AssertionError("no pattern found")


def _diagonal(d):
    import delfem2_gb300 as D
    K = D.CMatrixSparse()
    K.Initialize(d.size, 1, True)
    K.SetPattern(np.zeros(d.size + 1, np.uint32), np.zeros(0, np.uint32))
    K.set_values(np.zeros(0), d)
    return K


@pytest.mark.parametrize("n", [1024, 4096, 5120, 60_000, 400_000])
@pytest.mark.parametrize("above", [False, True])
def test_residual_norm_is_summed_in_fp64(gpu, n, above):
    import delfem2_gb300 as D
    b4, tol = _pattern(n, above)
    K, ilu = _diagonal(np.tile(D4, n // 4)), D.CPreconditionerILU()
    ident = _diagonal(np.ones(n))
    ilu.SetPattern0(ident)
    ilu.CopyValue(ident)
    assert ilu.Decompose()
    st = D.Solve_PCG_Mixed(np.tile(b4, n // 4), np.zeros(n), 1e-300, K, ilu, inner_tol=float(tol), max_iter=2,
                           max_outer=1, allow_not_converged=True)
    assert st.iterations == (1 if above else 2)  # the FP64 sum is below the tolerance: one iteration
