"""FP64 products whose chains run partly on the integer pipes (int_fma8 in
csrc/kernels.cuh) against the oracle's sequential chains, bit for bit: sizes
with more warps than the fed form takes, and values that meet its refusals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M, N, D, WIDTH = 701, 131, 733, 260  # 131 x 23 (22) column tiles, ragged in every size


def _values(kind, rng, n):
    if kind == "gauss":  # Poisson-like bands: binades change on the way up, hardly after the peak
        z = (np.arange(n) % WIDTH - WIDTH / 2) / 16.0
        return np.exp(-0.5 * z * z) * rng.uniform(0.5, 1.0, n)
    if kind == "powers":  # ties at the accumulator's grid, sums at the binades' ends
        return 2.0 ** -rng.integers(0, 56, n).astype(float)
    if kind == "signed":  # refused: the integer steps take b >= 0
        return rng.standard_normal(n)
    if kind == "extreme":  # beyond the exponents taken, subnormals and zeros
        v = rng.random(n) * 10.0 ** rng.choice([-310.0, -200.0, -3.0, 0.0, 60.0], n)
        v[rng.random(n) < 0.2] = 0.0
        return v
    return 1.0 + 2.0 ** -52 * rng.integers(0, 4, n)  # "ones": products just above powers of two


@pytest.mark.parametrize("kind", ["gauss", "powers", "signed", "extreme", "ones"])
@pytest.mark.parametrize("xkind", ["positive", "signed", "sparse"])
def test_integer_steps_bitwise(built, kind, xkind):
    import pqdts_gb300 as pq
    from oracle.oracle import Oracle
    from pqdts_gb300.synth import Instance

    rng = np.random.default_rng(len(kind) + 10 * len(xkind))
    lo = np.round(np.linspace(0, M - WIDTH, D)).astype(np.int64)
    inst = Instance(M, N, D, 0.0, 1e-6, lo, lo + WIDTH - 1, _values(kind, rng, D * WIDTH), rng.random((D, N)))
    X = rng.random((M, N)) if xkind == "positive" else rng.standard_normal((M, N)) * 10.0 ** rng.uniform(-9, 0, (M, N))
    if xkind == "sparse":
        X[rng.random((M, N)) < 0.5] = 0.0
        X[::5] = np.abs(X[::5]) * 2.0 ** rng.integers(-40, 3, X[::5].shape)
    if kind == "powers":
        X = np.where(X == 0, 0.0, np.sign(X) * 2.0 ** np.round(np.log2(np.abs(X) + 1e-300)))
    X = np.asfortranarray(X)
    o = Oracle.from_instance(inst)
    o.set_space(True, None)
    with pq.Solver(0) as s:
        s.set_instance(inst)
        s.set_x(X)
        assert np.array_equal(s.redO(), o.redO(X))
        assert np.array_equal(s.BF(X), o.BF(X))
